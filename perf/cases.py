"""The calls whose speed matters to a user of this package, as measurable cases.

listed() holds one case per kind of use: gradient flows (the relaxation that
both driver programs spend their time in) from the smallest supported grid to
the largest, in both precisions and on sizes with the factors 3 and 5; one
evaluation of a field (spectrum, energy, gradient norm, and back); the blocks
of the eigensolver (Hessian products, preconditioner) and the eigensolver
itself; the saddle search; a batch of relaxations of mixed sizes. draw(rng)
gives further cases of the same ranges.

Every case goes through spmiqc.SpmContext (or spmiqc.batch_grad_flow), the
Python mirror of the C ABI. Fields are sums of cosines over a shell of wave
vectors with |k| near 1, where the pair kernel has its minimum, plus noise:
what the drivers and the serving and batched workloads start from.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("spm-iqc_b200"))

import inputs  # noqa: E402
import spmiqc  # noqa: E402
import workloads  # noqa: E402

GAMMA, DT = 0.30, 0.3
SIZES = (32, 64, 96, 128, 160, 192, 256)


def listed():
    return [
        # a few steps on the smallest grid: the smoke run; launches and latency
        {"name": "flow_f64_n32", "kind": "flow", "N": 32, "prec": "fp64", "steps": 8, "L": 26.0, "Tau": -0.0061,
         "tuned": False},
        # the reference-sized relaxation: 500 steps at 64^3
        {"name": "flow_f64_n64", "kind": "flow", "N": 64, "prec": "fp64", "steps": 500, "L": 26.0, "Tau": -0.0061,
         "tuned": False},
        # FP32 phase of a mixed relaxation on a grid with the factor 3
        {"name": "flow_f32_n96", "kind": "flow", "N": 96, "prec": "fp32", "steps": 60, "L": 22.5, "Tau": -0.012,
         "tuned": False},
        # a grid with the factor 5, as in the batched relaxations
        {"name": "flow_f64_n160", "kind": "flow", "N": 160, "prec": "fp64", "steps": 40, "L": 19.0, "Tau": -0.003,
         "tuned": False},
        # the headline: gradient steps at 256^3, schedule tuned beforehand as a long run does
        {"name": "flow_f64_n256", "kind": "flow", "N": 256, "prec": "fp64", "steps": 50, "L": 26.0, "Tau": -0.0061,
         "tuned": True},
        # its FP32 phase
        {"name": "flow_f32_n256", "kind": "flow", "N": 256, "prec": "fp32", "steps": 50, "L": 26.0, "Tau": -0.0061,
         "tuned": True},
        # one look at a field: spectrum, energy, gradient with its norm, and the inverse transform
        {"name": "eval_f64_n192", "kind": "eval", "N": 192, "prec": "fp64", "L": 26.0, "Tau": -0.0061},
        # the eigensolver's block of Hessian products at the largest grid
        {"name": "hv_f64_n256_k8", "kind": "hv", "N": 256, "prec": "fp64", "nb": 8, "L": 26.0, "Tau": -0.0061},
        # its preconditioner on an odd-sized FP32 block
        {"name": "precond_f32_n128_k5", "kind": "precond", "N": 128, "prec": "fp32", "nb": 5, "L": 26.0,
         "Tau": -0.0061},
        # the lowest eight eigenpairs: four iterations from a random block
        {"name": "lobpcg_f64_n128_k8", "kind": "lobpcg", "N": 128, "prec": "fp64", "nb": 8, "iters": 4, "L": 26.0,
         "Tau": -0.0061},
        # saddle search: spring-pair iterations of two replicas
        {"name": "spm_f64_n192", "kind": "spm", "N": 192, "prec": "fp64", "iters": 6, "L": 26.0, "Tau": -0.0061},
        # many relaxations at once, two of each of three sizes
        {"name": "batch_f64_n64_n96_n128", "kind": "batch", "N": 128, "prec": "fp64", "sizes": "64,96,128,64,96,128",
         "steps": 64, "L": 24.0, "Tau": -0.01},
    ]


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "eval", "hv", "precond", "lobpcg", "spm", "batch"])
    N = rng.choice(SIZES)
    case = {"kind": kind, "N": N, "prec": rng.choice(["fp64", "fp32"]), "L": round(rng.uniform(18.0, 30.0), 3),
            "Tau": round(rng.uniform(-0.02, 0.0), 5)}
    cost = 256 ** 3 * 50  # points x steps of the largest listed case

    def spread(lo, hi):  # whole numbers, evenly over their logarithm
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    if kind == "flow":
        case["steps"] = spread(1, min(500, cost // N ** 3))
        case["tuned"] = N >= 192
    elif kind in ("hv", "precond"):
        case["nb"] = spread(1, 8)
    elif kind == "lobpcg":
        case.update(N=rng.choice([32, 64, 96, 128]), prec="fp64", nb=rng.randint(2, 8), iters=rng.randint(2, 4))
    elif kind == "spm":
        case.update(prec="fp64", iters=spread(1, max(1, min(12, cost // (10 * N ** 3)))))
    elif kind == "batch":
        sizes = [rng.choice([32, 64, 96, 128, 160]) for _ in range(rng.randint(2, 8))]
        case.update(N=max(sizes), sizes=",".join(str(n) for n in sizes), steps=spread(16, 64))
    return case


# ------------------------------------------------------------------ inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _field(N, L, seed, amp=0.15):
    """A BCC-shell cosine field of rms amp with 1e-3 noise (FP64, on the GPU)."""
    vec = workloads.shell_vectors("bcc", L)
    while np.max(np.abs(vec)) >= N // 2:  # a shell beyond the grid's range is halved until it fits
        vec = np.unique(np.round(vec / 2.0).astype(np.int64), axis=0)
        vec = vec[np.any(vec != 0, axis=1)]
    theta = 2 * np.pi * inputs.unit(seed, np.arange(len(vec), dtype=np.uint64))
    i = torch.arange(N, device=_device(), dtype=torch.float64) * (2 * math.pi / N)
    phi = torch.zeros((N, N, N), device=_device(), dtype=torch.float64)
    for n, th in zip(vec, theta):
        plane = float(n[0]) * i[:, None] + float(n[1]) * i[None, :] + float(th)
        kz = float(n[2]) * i
        phi += torch.cos(plane)[:, :, None] * torch.cos(kz) - torch.sin(plane)[:, :, None] * torch.sin(kz)
    phi *= amp * math.sqrt(2.0 / len(vec))
    phi += 1e-3 * torch.randn((N, N, N), device=_device(), dtype=torch.float64, generator=_gen(seed))
    return phi - phi.mean()


def _inputs(case, seed):
    """The case's input fields in its precision, from the seed alone."""
    N, L, kind = case["N"], case["L"], case["kind"]
    dtype = torch.float64 if case["prec"] == "fp64" else torch.float32
    if kind == "batch":
        return {"phi": [_field(int(n), L, seed * 64 + j).to(dtype) for j, n in enumerate(case["sizes"].split(","))]}
    got = {"phi": _field(N, L, seed).to(dtype)}
    if kind in ("hv", "precond"):
        got["v"] = torch.randn((case["nb"], N, N, N), device=_device(), dtype=dtype, generator=_gen(seed + 7919))
    elif kind == "spm":  # a long-wavelength displacement along x, as the saddle-search jobs start with
        d = torch.cos(2 * math.pi * (1 + seed % 3) * torch.arange(N, device=_device(), dtype=torch.float64) / N)
        got["phi1"] = got["phi"] + 0.01 * d[:, None, None].to(dtype)
    return got


def _context(case, N=None):
    return spmiqc.SpmContext(N or case["N"], case["L"], case["Tau"], GAMMA, DT, case["prec"])


def prepare(case, seed):
    state = {"case": case, **_inputs(case, seed)}
    kind = case["kind"]
    if kind == "batch":
        state["ctx"] = [_context(case, p.shape[0]) for p in state["phi"]]
        state["work"] = [(c.field(), c.spectrum()) for c in state["ctx"]]
        return state
    ctx = state["ctx"] = _context(case)
    if kind == "flow":
        if case["tuned"]:
            ctx.autotune(20)
        state["work"] = (ctx.field(), ctx.spectrum())
    elif kind == "eval":
        state["work"] = (ctx.spectrum(), ctx.field(), ctx.field())
    elif kind in ("hv", "precond"):
        state["out"] = torch.empty_like(state["v"])
    elif kind == "lobpcg":
        state["v"] = ctx.hiosd_lobpcg_initialization(case["nb"], seed)
        state["out"] = torch.empty_like(state["v"])
    elif kind == "spm":
        state["work"] = (ctx.field(), ctx.field())
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "flow":  # a relaxation from an initial field: its spectrum, then the steps
        phi, uh = state["work"]
        phi.copy_(state["phi"])
        ctx.my_fft(phi, uh)
        return {"stats": ctx.get_min_u_F(phi, uh, case["steps"]), "phi": phi, "uhat": uh}
    if kind == "batch":
        for c, p0, (p, u) in zip(ctx, state["phi"], state["work"]):
            p.copy_(p0)
            c.my_fft(p, u)
        torch.cuda.current_stream().synchronize()
        done = spmiqc.batch_grad_flow(ctx, [p for p, _ in state["work"]], [u for _, u in state["work"]],
                                      case["steps"], 1e-12)
        return {"steps": done, "phi": [p for p, _ in state["work"]], "uhat": [u for _, u in state["work"]]}
    if kind == "eval":
        uh, grad, back = state["work"]
        ctx.my_fft(state["phi"], uh)
        energy = ctx.get_Ene(state["phi"], uh)
        _, norm = ctx.ngrad_cam(state["phi"], grad)
        ctx.my_ifft(uh, back)
        return {"uhat": uh, "energy": energy, "grad": grad, "norm": norm, "back": back}
    if kind == "hv":
        return ctx.hv_cam(state["phi"], state["v"], state["out"])
    if kind == "precond":
        state["out"].copy_(state["v"])
        return ctx.precond_camnew(state["out"])
    if kind == "lobpcg":
        state["out"].copy_(state["v"])
        ev, res, _ = ctx.hiosd_lobpcg_inip(state["phi"], state["out"], case["iters"])
        return {"evals": ev, "resid": res, "V": state["out"]}
    a, b = state["work"]
    a.copy_(state["phi"])
    b.copy_(state["phi1"])
    return {"res": ctx.Spring_Pairing(a, b, case["iters"], 1e-14), "phi0": a, "phi1": b}


# ------------------------------------------------------------------ work
def work(case):
    N, kind = case["N"], case["kind"]
    es = 8 if case["prec"] == "fp64" else 4

    def fft(n):  # a real-to-complex or complex-to-real transform
        return 2.5 * n ** 3 * math.log2(n ** 3)

    def flow(n, steps):  # one transform, then two a step and about 30 operations a point
        return {"bytes": 3 * es * n ** 3, "flops": fft(n) + steps * (2 * fft(n) + 30.0 * n ** 3)}

    S, F = es * N ** 3, fft(N)
    if kind == "flow":
        return flow(N, case["steps"])
    if kind == "batch":
        parts = [flow(int(n), case["steps"]) for n in case["sizes"].split(",")]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "eval":
        return {"bytes": 4 * S, "flops": 4 * F + 40.0 * N ** 3}
    if kind == "hv":
        return {"bytes": (1 + 2 * case["nb"]) * S, "flops": case["nb"] * (2 * F + 10.0 * N ** 3)}
    if kind == "precond":
        return {"bytes": 2 * case["nb"] * S, "flops": case["nb"] * (2 * F + 4.0 * N ** 3)}
    if kind == "lobpcg":  # 3k products and k preconditioners an iteration, a 3k x 3k Gram, updates
        k = case["nb"]
        return {"bytes": (1 + 2 * k) * S,
                "flops": case["iters"] * (k * (8 * F + 34.0 * N ** 3) + 50.0 * k * k * N ** 3)}
    return {"bytes": 4 * S, "flops": case["iters"] * (16 * F + 120.0 * N ** 3)}


# ------------------------------------------------------------------ 64-bit values
class _Model:
    """The model's routines in plain FP64 torch on the R2C half spectrum."""

    def __init__(self, N, L, Tau):
        self.N, self.n3, self.Tau = N, float(N) ** 3, Tau
        k = torch.fft.fftfreq(N, d=1.0 / N, device=_device(), dtype=torch.float64)
        kz = torch.arange(N // 2 + 1, device=_device(), dtype=torch.float64)
        k2 = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz ** 2) / (L * L)
        poly = 1.969182919080340 + k2 * (-14.949858723012090 + k2 * (
            37.445683882581790 + k2 * (-38.839451762550148 + k2 * 13.999261011773505)))
        self.G = torch.exp(-0.5 * k2 / 0.568809 ** 2) * poly + 0.08
        self.w = torch.full((N // 2 + 1,), 2.0, device=_device(), dtype=torch.float64)
        self.w[0] = self.w[-1] = 1.0

    def fft(self, x):
        return torch.fft.rfftn(x) / self.n3

    def ifft(self, X):
        return torch.fft.irfftn(X, s=(self.N,) * 3) * self.n3

    def packed(self, X):
        P = X[..., :-1].clone()
        P[..., 0] += 1j * X[..., -1]
        return P

    def force(self, x):
        return x * (self.Tau + x * (GAMMA - x))

    def e2(self, x):
        return float((x * x * (-0.5 * self.Tau + x * (-GAMMA / 3 + 0.25 * x))).mean())

    def e1(self, X):
        return 0.5 * float((self.w * self.G * (X.real ** 2 + X.imag ** 2)).sum())

    def flow(self, phi, steps):
        u, stats = self.fft(phi), []
        for _ in range(steps):
            f = self.fft(self.force(phi))
            u1 = (DT * f + u) / (1 + DT * self.G)
            u1[0, 0, 0] = 0
            g = self.G * u - f
            g[0, 0, 0] = 0
            e1 = self.e1(u)
            stats.append([e1 + self.e2(phi), float((u1.real - u.real).abs().max()),
                          math.sqrt(float((self.w * (g.real ** 2 + g.imag ** 2)).sum())), e1])
            u, phi = u1, self.ifft(u1)
        return phi, self.packed(u), np.array(stats).reshape(-1, 4)

    def ngrad(self, phi):
        X = self.fft(phi) * self.G
        X[0, 0, 0] = 0
        g = self.force(phi) - self.ifft(X)
        return g - g.mean()

    def hv(self, phi, v):
        h = self.ifft(self.fft(v) * self.G) + (-self.Tau - 2 * GAMMA * phi + 3 * phi * phi) * v
        return h - h.mean()

    def precond(self, w):
        w = self.ifft(self.fft(w) / (self.G + abs(self.Tau) + 0.02))
        return w - w.mean()

    def tangent(self, a, b):
        return (b - a) / math.sqrt(float(((b - a) ** 2).mean()))

    def force_step(self, x, v, factor):
        s = factor * float((self.ngrad(x) * v).mean())
        X = self.fft(x + self.force(x) - s * v) / (1 + self.G)
        X[0, 0, 0] = 0
        return self.ifft(X)

    def spring_pairing(self, a, b, iters):
        P, hist = [a, b], []

        def spring():
            P[0] = P[0] + 0.001 * (P[1] - P[0])
            P[1] = P[1] + 0.001 * (P[0] - P[1])

        for _ in range(iters):
            v = self.tangent(*P)
            P[:] = [self.force_step(p, v, 1.0) for p in P]
            spring()
            v = self.tangent(*P)
            P[:] = [self.force_step(p, v, 2.0) for p in P]
            hist.append(max(math.sqrt(float((self.ngrad(p) ** 2).mean())) for p in P))
            spring()
        return np.array(hist), P[0], P[1]


def exact(case, seed):
    kind = case["kind"]
    if kind == "lobpcg":  # the iterates of a random block have no value to compare with
        return None
    x = _inputs(case, seed)
    if kind == "batch":
        got = [_Model(p.shape[0], case["L"], case["Tau"]).flow(p.double(), case["steps"]) for p in x["phi"]]
        return {"steps": None, "phi": [g[0] for g in got], "uhat": [g[1] for g in got]}
    m = _Model(case["N"], case["L"], case["Tau"])
    phi = x["phi"].double()
    if kind == "flow":
        phi, uh, stats = m.flow(phi, case["steps"])
        return {"stats": stats, "phi": phi, "uhat": uh}
    if kind == "eval":
        X, g = m.fft(phi), m.ngrad(phi)
        return {"uhat": m.packed(X), "energy": m.e1(X) + m.e2(phi), "grad": g,
                "norm": math.sqrt(float((g * g).mean())), "back": phi}
    if kind == "hv":
        return torch.stack([m.hv(phi, v.double()) for v in x["v"]])
    if kind == "precond":
        return torch.stack([m.precond(v.double()) for v in x["v"]])
    hist, a, b = m.spring_pairing(phi, x["phi1"].double(), case["iters"])
    return {"res": hist, "phi0": a, "phi1": b}
