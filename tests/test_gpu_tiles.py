"""The tile passes (tile_kernels.cuh) at every grid size against the NumPy
oracle: Hessian-product and preconditioner blocks in both precisions, and a
gradient chain that stops inside (its tile-ordered spectrum goes back to the
caller's array).

Bars: FP64 1e-11 of the largest value (the parity bar of the other tests).
FP32: a transform pair of N^3 points rounds each value about 2 log2(N^3) times;
with errors of at most eps = 2^-24 per rounding and operands up to ~6 rms (a
unit-variance random block) the bar is 6 * 2 * 3 log2(N) * 2^-24 of the rms,
at most 1.8e-5 (N = 256)."""
import numpy as np
import pytest

from conftest import rel
from oracle import spmiqc_np as npo

pytestmark = pytest.mark.gpu

SIZES = [32, 64, 96, 128, 160, 192, 256]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("N", SIZES)
def test_blocks_match_oracle(cuda, N, prec):
    import spmiqc
    m = npo.Model(N, L=21.3, Tau=-0.013)
    c = spmiqc.SpmContext(N, L=21.3, Tau=-0.013, precision=prec)
    dt = np.float64 if prec == "fp64" else np.float32
    rng = np.random.default_rng(N)
    phi = (0.1 * rng.standard_normal((N, N, N))).astype(dt)
    nb = 1 if N == 256 else 3
    v = rng.standard_normal((nb, N, N, N)).astype(dt)
    v[0] += dt(0.5)  # a mean, so the k = 0 modes matter
    vd = cuda.from_numpy(v).cuda()
    h = c.hv_cam(cuda.from_numpy(phi).cuda(), vd).cpu().numpy().astype(np.float64)
    w = c.precond_camnew(vd).cpu().numpy().astype(np.float64)
    for b in range(nb):
        x = v[b].astype(np.float64)
        for got, ref in ((h[b], m.hv(phi.astype(np.float64), x)), (w[b], m.precond(x))):
            if prec == "fp64":
                assert rel(got, ref) < 1e-11
            else:
                bar = 36 * np.log2(N) * 2.0 ** -24 * np.sqrt(np.mean(ref * ref))
                assert np.max(np.abs(got - ref)) < bar
    c.close()


@pytest.mark.parametrize("N", SIZES)
def test_chain_stopping_inside_returns_its_state(cuda, N):
    """A flow that reaches tol_grad inside an enqueued chain leaves phi and uhat
    of its last step: uhat = my_fft(phi), and both as a flow of exactly that
    many steps gives them."""
    import spmiqc
    phi0 = npo.uniform_field(N, 77)
    ctx = spmiqc.SpmContext(N, Tau=-0.02)

    def flow(steps, tol):
        p = cuda.from_numpy(phi0.copy()).cuda()
        u = ctx.my_fft(p)
        return ctx.get_min_u_F(p, u, steps, tol_grad=tol), p, u

    probe, _, _ = flow(30, 0.0)
    st, p, u = flow(400, float(probe[19, 2]))  # reached at step 20, inside the second chunk
    assert len(st) == 20
    _, q, w = flow(20, 0.0)
    assert cuda.equal(p, q) and cuda.equal(u, w)
    back = ctx.my_fft(p)
    assert rel(back.cpu().numpy(), u.cpu().numpy()) < 1e-11
    ctx.close()


@pytest.mark.parametrize("N", SIZES)
def test_energy_matches_oracle(cuda, N):
    """get_Ene streams the field and the packed spectrum (its c = 0 column
    unpacked with partner rows). Bar: a few roundings a term and a tree of sums,
    2^-53 * 40 log2(N^3) < 1.1e-13 of the terms' absolute sum, which is at most ten times
    the energy for this field: 1e-12."""
    import spmiqc
    m = npo.Model(N, L=19.7, Tau=-0.05)
    c = spmiqc.SpmContext(N, L=19.7, Tau=-0.05)
    phi = npo.uniform_field(N, 5, amp=0.4)
    pd = cuda.from_numpy(phi).cuda()
    e, ref = c.get_Ene(pd, c.my_fft(pd)), m.energy(phi, m.my_fft(phi))
    assert abs(e - ref) < 1e-12 * abs(ref)
    c.close()


def test_many_groups_run_through_a_graph(cuda):
    """Nine instances with launches of their own (batch_group 0) go through the
    captured graph, the same nine in one group are launched directly: the same
    steps and fields."""
    import spmiqc
    out = []
    for group in (0, 1):
        cs = [spmiqc.SpmContext(32, L=18.0 + i, Tau=-0.002 * i) for i in range(9)]
        for c in cs:
            c.tune("batch_group", group)
        ps = [cuda.from_numpy(npo.uniform_field(32, 100 + i)).cuda() for i in range(9)]
        us = [c.my_fft(p) for c, p in zip(cs, ps)]
        cuda.cuda.synchronize()
        out.append((spmiqc.batch_grad_flow(cs, ps, us, 70, 1e-12, steps_per_launch=16), ps, us))
        for c in cs:
            c.close()
    (d0, p0, u0), (d1, p1, u1) = out
    assert d0 == d1 == [70] * 9
    for a, b in zip(p0 + u0, p1 + u1):
        assert cuda.equal(a, b)


@pytest.mark.parametrize("K", [16, 50])
def test_floor_detection_does_not_depend_on_the_launch_path(cuda, K):
    """Mixed batches whose FP32 phase ends at its rounding floor, between rounds of K
    steps: launched directly (one group) or through the graph (nine), an instance
    hands over to FP64 after the same step, with the same counts and fields."""
    import spmiqc
    out = []
    for group in (0, 1):
        cs = [spmiqc.SpmContext(32, L=18.0 + i, Tau=0.5 - 0.002 * i) for i in range(9)]
        for c in cs:
            c.tune("batch_group", group)
        ps = [cuda.from_numpy(npo.uniform_field(32, 100 + i)).cuda() for i in range(9)]
        us = [c.my_fft(p) for c, p in zip(cs, ps)]
        cuda.cuda.synchronize()
        out.append((spmiqc.batch_grad_flow(cs, ps, us, 12000, 1e-10, 1e-9, steps_per_launch=K), ps, us))
        for c in cs:
            c.close()
    (d0, p0, u0), (d1, p1, u1) = out
    assert d0 == d1
    for a, b in zip(p0 + u0, p1 + u1):
        assert cuda.equal(a, b)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("N", [32, 64, 128])
def test_operations_in_a_row_read_what_the_one_before_wrote(cuda, N, prec):
    """Grids of one wave are launched while the launch before still runs. Operations
    in a row, each on the fields that the one before has just written (tangent,
    force steps along it, a Hessian product, a preconditioner, transforms and a
    flow), give the same bits as with the device idle in between."""
    import spmiqc
    dt = np.float64 if prec == "fp64" else np.float32
    c = spmiqc.SpmContext(N, Tau=-0.02, precision=prec)
    a, b = (cuda.from_numpy(npo.uniform_field(N, s).astype(dt)).cuda() for s in (3, 4))
    out = []
    for idle in (False, True):
        got = []

        def did(x):
            got.append(x)
            if idle:
                cuda.cuda.synchronize()
            return x

        x = did(a.clone())
        for _ in range(4):
            v = did(c.get_Tv(x, b))
            did(c.Natural_Forces(x, v))
            did(c.MinMax_Forces(x, v))
            h = did(c.hv_cam(x, v))
            did(c.precond_camnew(h))
            x = did(x + 0.01 * h)  # small: the flow below stays stable
            did(c.get_Tv(v, x, h))
            u = did(c.my_fft(x))
            did(c.my_ifft(u, x))
            c.get_min_u_F(x, u, 3)
        cuda.cuda.synchronize()
        out.append([t.clone() for t in got])
    for p, q in zip(*out):
        assert cuda.equal(p, q)
    c.close()


@pytest.mark.parametrize("ng,steps,graph", [(2, 176, False), (2, 192, True), (8, 32, False), (8, 48, True),
                                            (1, 496, False), (1, 512, True)])
def test_long_batches_of_several_groups_take_the_graph(cuda, ng, steps, graph):
    """Groups that share no launch (batch_group 0) are launched from one host thread:
    over 24 / ng rounds or more (32 for one group) they go through the captured graph, whose
    launches the host issues once. The host's launches tell the ways apart (a step takes two,
    a captured one is counted once), and fields and counts are those of a plain flow."""
    import spmiqc
    K = 16
    cs = [spmiqc.SpmContext(32, L=18.0 + i) for i in range(ng)]
    for c in cs:
        c.tune("batch_group", 0)
    start = [npo.uniform_field(32, 200 + i) for i in range(ng)]
    ps = [cuda.from_numpy(x.copy()).cuda() for x in start]
    us = [c.my_fft(p) for c, p in zip(cs, ps)]
    cuda.cuda.synchronize()
    count = spmiqc.lib().spm_launch_count
    before = [count(c.h) for c in cs]
    assert spmiqc.batch_grad_flow(cs, ps, us, steps, 1e-14, steps_per_launch=K) == [steps] * ng
    for c, b in zip(cs, before):
        # one step ahead and one captured round, or every round
        assert (count(c.h) - b < 4 * K) == graph
    for c, x, p, u in zip(cs, start, ps, us):
        q = cuda.from_numpy(x).cuda()
        w = c.my_fft(q)
        c.get_min_u_F(q, w, steps)
        assert cuda.equal(p, q) and cuda.equal(u, w)
        c.close()


@pytest.mark.parametrize("n", [2, 9])
def test_refused_batch_gives_its_contexts_back(cuda, n):
    """A batch whose last spectrum is not 16-byte aligned is refused after its streams
    exist, launched directly (2 groups) or on the way to the graph (9): the contexts
    run on their own stream again, without the batch's limits."""
    import spmiqc
    N = 32
    cs = [spmiqc.SpmContext(N, L=18.0 + i) for i in range(n)]
    for c in cs:
        c.tune("batch_group", 0)
    start = [npo.uniform_field(N, 300 + i) for i in range(n)]
    ps = [cuda.from_numpy(x.copy()).cuda() for x in start]
    us = [c.my_fft(p) for c, p in zip(cs, ps)]
    odd = cuda.zeros(N ** 3 + 1, dtype=cuda.float64, device="cuda")[1:]
    cuda.cuda.synchronize()
    with pytest.raises(spmiqc.SpmError) as err:
        spmiqc.batch_grad_flow(cs, ps, us[:-1] + [odd], 64, 1e30)
    assert err.value.status == spmiqc.SPM_ERR_ARG
    for c, x in zip(cs, start):
        m = npo.Model(N, L=c.L)
        q = cuda.from_numpy(x.copy()).cuda()
        u = c.my_fft(q)
        assert rel(c.to_full(u).cpu().numpy(), m.my_fft(x)) < 1e-11
        assert len(c.get_min_u_F(q, u, 5)) == 5
        c.close()


def test_autotuned_choice_does_not_depend_on_the_first_context(cuda):
    """The remembered FP64 choice comes from fixed candidates: a first context with
    the fused plane pass off (a store and a load of phi more a step) does not switch it
    off for later ones. The knobs that FP64 kernels do not read stay the caller's."""
    import spmiqc
    N = 160
    c = spmiqc.SpmContext(N)
    c.tune("fuse_planes", 0)
    c.tune("plane_cps", 3)
    c.autotune(20)
    assert c.tuning()["fuse_planes"] == 1 and c.tuning()["plane_cps"] == 3
    d = spmiqc.SpmContext(N)
    d.autotune(20)
    assert d.tuning()["fuse_planes"] == 1 and d.tuning()["plane_cps"] == 2
    assert d.tuning()["pdl"] == c.tuning()["pdl"]
    c.close()
    d.close()


def test_autotuning_a_context_tunes_its_fp32_twin(cuda):
    """spm_autotune on an FP64 context chooses the schedule of the FP32 twin that its
    mixed flows run on, as it does for an FP32 context; knobs set afterwards win."""
    import spmiqc
    N = 128
    names = ("plane_cps", "fuse_planes", "plane_xg", "pencil_tc", "pdl")
    get = spmiqc.lib().spm_tune_get
    get.argtypes = [spmiqc.ctypes.c_void_p, spmiqc.ctypes.c_char_p]

    def twin(c):
        return {k: int(get(c.h, ("twin_" + k).encode())) for k in names}

    c = spmiqc.SpmContext(N)
    c.autotune(20)
    got = twin(c)
    assert (got["plane_cps"], got["plane_xg"]) in {(1, 0), (2, 0), (3, 0), (2, 1), (2, 2), (2, 3), (3, 3), (4, 3),
                                                   (5, 3), (6, 3)}
    d = spmiqc.SpmContext(N, precision="fp32")
    d.autotune(20)  # the same search, remembered
    assert d.tuning() == {k: got[k] for k in d.tuning()}
    # the mixed flow runs with it: the records of an FP32 context of that schedule
    phi = npo.uniform_field(N, 8)
    p = cuda.from_numpy(phi.copy()).cuda()
    st, n32, n64 = c.get_min_u_F_mixed(p, c.my_fft(p), 30, 1e-14, 1e-13)
    q = cuda.from_numpy(phi).cuda()
    u = c.my_fft(q)
    q32, u32 = q.float(), cuda.view_as_real(u).float() if u.is_complex() else u.float()
    assert (n32, n64) == (30, 0)
    assert np.array_equal(st, d.get_min_u_F(q32, u32, 30))
    e = spmiqc.SpmContext(N)
    e.autotune(20)
    assert e.tuning() == c.tuning() and twin(e) == got
    c.close()
    d.close()
    e.close()


def test_knobs_set_after_tuning_win_over_the_twins_choice(cuda):
    import spmiqc
    N = 96  # (no FP32 context of this size is tuned here: its choice would win)
    get = spmiqc.lib().spm_tune_get
    get.argtypes = [spmiqc.ctypes.c_void_p, spmiqc.ctypes.c_char_p]
    c = spmiqc.SpmContext(N)
    c.autotune(20)
    for cps in (1, 3):
        c.tune("plane_cps", cps)
        assert get(c.h, b"twin_plane_cps") == cps == c.tuning()["plane_cps"]
    c.autotune(20)
    assert get(c.h, b"twin_plane_cps") >= 1 and c.tuning()["plane_cps"] == 3
    assert get(c.h, b"twin_nothing") == -1
    c.close()


def test_steps_of_extreme_size(cuda):
    """The step factor 1 / (1 + dt G) beyond the smallest normal number. Both dt = 1e300
    and dt = 8e307 (denominators up to 1.6e308, factors down to 6e-309) give the
    spectrum f / G, on the same G (its least value, 2.8e-7, is known to 1e-10 only, so
    the oracle's is another): they differ by the rounding of the factors, a subnormal
    number of at least 49 bits, of products, and of the inverse transform, 2^-49 + 30 * 2^-52 < 1e-13
    of the largest value. A tiny dt leaves the field as it is."""
    import spmiqc
    N = 32
    phi = npo.uniform_field(N, 9)
    got = {}
    for dt in (1e300, 8e307, 1e-300):
        c = spmiqc.SpmContext(N, dt=dt)
        p = cuda.from_numpy(phi.copy()).cuda()
        st = c.get_min_u_F(p, c.my_fft(p), 1)
        assert len(st) == 1 and np.all(np.isfinite(st))
        got[dt] = p.cpu().numpy()
        c.close()
    assert np.max(np.abs(got[1e300])) > 1
    assert rel(got[8e307], got[1e300]) < 1e-13
    assert rel(got[1e-300], phi - phi.mean()) < 1e-13


def test_preconditioner_with_an_extreme_tau(cuda):
    """1 / (G + |Tau| + 0.02) with Tau beyond 2^1022, where it is a subnormal number of 50
    bits: on a field of 1e300 the result is w / Tau minus its mean, to the 1e-13 of the
    step above."""
    import spmiqc
    N = 32
    w = npo.uniform_field(N, 12, amp=1e300)
    c = spmiqc.SpmContext(N, Tau=-1e308)
    got = c.precond_camnew(cuda.from_numpy(w.copy()).cuda()).cpu().numpy()
    ref = w / 1e308
    assert rel(got, ref - ref.mean()) < 1e-13
    c.close()


def test_block_of_two_at_the_largest_grid(cuda):
    """256^3 FP64 is where the plane passes copy their tiles through a stage, with a
    tensor map per field: two different vectors against the oracle, and each alone."""
    import spmiqc
    N = 256
    m = npo.Model(N, L=21.3, Tau=-0.013)
    c = spmiqc.SpmContext(N, L=21.3, Tau=-0.013)
    rng = np.random.default_rng(11)
    phi = 0.1 * rng.standard_normal((N, N, N))
    v = rng.standard_normal((2, N, N, N))
    v[1] += 0.25
    pd, vd = cuda.from_numpy(phi).cuda(), cuda.from_numpy(v).cuda()
    h = c.hv_cam(pd, vd)
    for b in range(2):
        assert cuda.equal(c.hv_cam(pd, vd[b]), h[b])
        assert rel(h[b].cpu().numpy(), m.hv(phi, v[b])) < 1e-11
    w = c.precond_camnew(vd).cpu().numpy()
    for b in range(2):
        assert rel(w[b], m.precond(v[b])) < 1e-11
    c.close()


@pytest.mark.parametrize("pdl", [0, 1])
@pytest.mark.parametrize("N", [32, 96, 160, 192])
def test_fields_alone_and_in_a_block_fused_and_not(cuda, N, pdl):
    """What acts on the FP64 passes: the number of fields in a launch (single-wave grids
    let the next launch in, several fields may not), dependent launches, and the joint
    plane pass. The same bits."""
    import spmiqc
    phi = npo.uniform_field(N, 21)
    V = cuda.from_numpy(np.stack([npo.uniform_field(N, 70 + i, amp=1.0) for i in range(3)])).cuda()
    out = []
    for fuse in (0, 1):
        c = spmiqc.SpmContext(N, Tau=-0.02)
        c.tune("pdl", pdl)
        c.tune("fuse_planes", fuse)
        p = cuda.from_numpy(phi.copy()).cuda()
        u = c.my_fft(p)
        st = c.get_min_u_F(p, u, 11)
        h = c.hv_cam(p, V)
        w = c.precond_camnew(V.clone())
        for b in range(3):
            assert cuda.equal(c.hv_cam(p, V[b]), h[b])
            assert cuda.equal(c.precond_camnew(V[b].clone()), w[b])
        out.append((st, p, u, h, w))
        c.close()
    (s0, *a), (s1, *b) = out
    assert np.array_equal(s0, s1) and all(cuda.equal(x, y) for x, y in zip(a, b))
