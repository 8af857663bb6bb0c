// Kernel chains of each hot-path routine for one grid size N and real type T.
// Instantiated once per (N, T) in inst_<N>.cu; the host API reaches them
// through the OpsTable of the context.
#pragma once

#include <algorithm>

#include "cluster_impl.cuh"
#include "launch.cuh"
#include "tile_kernels.cuh"

namespace spm {

// Persistent launch of a tile kernel: as many blocks as can be resident at once
// (queried once per kernel and device), at most one per tile, for each of nb
// fields. The grid depends only on the kernel and the device (never on the
// load), so the reductions' partial sums, and hence the results, do not
// either. With pdl_on the launch is a programmatic dependent one: it may be set
// up while the previous kernel of the stream finishes, and waits for it in
// grid_dep_sync. Grids that are resident at once with a tile per block (plane
// passes up to 128^3, pencil passes up to 64^3) are launched that way in any
// case, and let the next launch in as soon as they run: its blocks are then
// placed, with their twiddles loaded, when this one completes.
template <class Tag, class K, class P>
static int launch_tiles(spm_ctx *c, K kern, int threads, size_t smem, int tiles, P &p, int nb, const char *what) {
  cudaError_t e = prepare<Tag>(kern, smem, c->device);
  if (e != cudaSuccess) return spm_fail_cuda(e, what);
  static std::atomic<int> resident[32] = {};
  const int dev = c->device < 32 ? c->device : 0;
  int most = resident[dev].load(std::memory_order_relaxed);
  if (most == 0) {
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    if (e != cudaSuccess || per_sm < 1)
      return spm_fail_cuda(e != cudaSuccess ? e : cudaErrorInvalidConfiguration, what);
    most = per_sm * sms;
    resident[dev].store(most, std::memory_order_relaxed);
  }
  const int nbk = std::min({most, tiles, kPartStride});
  p.trigger = nbk == tiles && nbk * nb <= most;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nb, nbk, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_on(c) || p.trigger ? 1 : 0;
  c->launches++;
  e = cudaLaunchKernelEx(&cfg, kern, p);
  return e == cudaSuccess ? 0 : spm_fail_cuda(e, what);
}

template <int N, class T, class Pro> static int plane_fwd(spm_ctx *c, KParams &p, int nb) {
  struct Tag {};
  return launch_tiles<Tag>(c, plane_fwd_kernel<N, T, Pro>, N, plane_smem<N, T>(), PlaneGeo<N, T>::TILES, p, nb,
                           "plane_fwd");
}
// The plane kernels that read the scratch: G groups of N threads per block, with
// the maps of their tensor copies for G > 1.
template <class Tag, int N, class T, class K> static int launch_inv(spm_ctx *c, K kern, const KParams &p, int nb,
                                                                    const char *what) {
  constexpr int G = inv_groups<N, T>();
  TileParams<G> q;
  static_cast<KParams &>(q) = p;
  if constexpr (G > 1)
    for (int b = 0; b < nb; b++) SPM_TRY(spm_scratch_map(c, p.in[b], &q.tm[b]));
  return launch_tiles<Tag>(c, kern, G * N, plane_smem<N, T, G>(), PlaneGeo<N, T>::TILES / G, q, nb, what);
}
template <int N, class T, class Epi> static int plane_inv(spm_ctx *c, const KParams &p, int nb) {
  struct Tag {};
  return launch_inv<Tag, N, T>(c, plane_inv_kernel<N, T, Epi>, p, nb, "plane_inv");
}
template <int N, class T, class Epi, class Pro> static int plane_inv_fwd(spm_ctx *c, const KParams &p, int nb) {
  struct Tag {};
  return launch_inv<Tag, N, T>(c, plane_inv_fwd_kernel<N, T, Epi, Pro>, p, nb, "plane_inv_fwd");
}
template <int N, class T, class Op> static int pencil(spm_ctx *c, KParams &p, int nb) {
  struct Tag {};
  using PG = PencilGeo<N, T>;
  if constexpr (Op::SI)
    for (int b = 0; b < nb; b++)
      if (((uintptr_t)p.st[b] & 15u) != 0) return spm_fail(SPM_ERR_ARG, "spectrum buffers must be 16-byte aligned");
  return launch_tiles<Tag>(c, pencil_kernel<N, T, Op>, PG::TH, pencil_smem<N, T>(), PG::TILES, p, nb, "pencil");
}

template <int N, class T> struct Impl {
  static int fft(spm_ctx *c, const void *x, void *xhat) {
    SPM_NEED_SCRATCH(c, 1);
    KParams p = spm_params(c);
    p.in[0] = x;
    p.out[0] = spm_buf(c, 0);
    SPM_TRY((plane_fwd<N, T, ProIdent<T>>(c, p, 1)));
    KParams q = spm_params(c);
    q.in[0] = spm_buf(c, 0);
    q.sto[0] = xhat;
    return pencil<N, T, OpFwd<T>>(c, q, 1);
  }

  static int ifft(spm_ctx *c, const void *xhat, void *x) {
    SPM_NEED_SCRATCH(c, 1);
    KParams q = spm_params(c);
    q.st[0] = xhat;
    q.out[0] = spm_buf(c, 0);
    SPM_TRY((pencil<N, T, OpInv<T>>(c, q, 1)));
    KParams p = spm_params(c);
    p.in[0] = spm_buf(c, 0);
    p.out[0] = x;
    return plane_inv<N, T, EpiStore<T>>(c, p, 1);
  }

  // E2 -> scal[SC_E2], E1 -> scal[SC_E1]
  static int energy(spm_ctx *c, const void *phi, const void *uhat) {
    if (((uintptr_t)uhat & 15u) != 0) return spm_fail(SPM_ERR_ARG, "spectrum buffers must be 16-byte aligned");
    KParams p = spm_params(c);
    p.in[0] = phi;
    p.st[0] = uhat;
    c->launches++;
    // blocks: eight per SM, or two, get_Ene with its read-back: 32^3 42.3 / 41.7, 64^3 and
    // 96^3 equal, 128^3 42.0 / 43.5, 192^3 65 / 91, 256^3 111 / 172 us
    energy_kernel<T><<<N >= 128 ? kReduceBlocks : kReduceBlocks / 4, kThreads, 0, c->stream>>>(p, N);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : spm_fail_cuda(e, "energy");
  }

  // One semi-implicit step of three passes, gated by the flow words. With ev
  // non-null, records ev[0..3] around the passes (for per-kernel timing).
  static int grad_step_ev(spm_ctx *c, void *phi, void *uhat, void *const *ev) {
    SPM_NEED_SCRATCH(c, 1);
    const Step s{&c, &phi, &uhat, 1};
    auto rec = [&](int i) {
      if (ev) cudaEventRecord((cudaEvent_t)ev[i], c->stream);
    };
    rec(0);
    SPM_TRY(s.head());
    rec(1);
    SPM_TRY(s.spectral(false, false));
    rec(2);
    SPM_TRY(s.tail());
    rec(3);
    return 0;
  }
  static int grad_step(spm_ctx *c, void *phi, void *uhat) { return grad_step_ev(c, phi, uhat, nullptr); }

  // The passes of a gradient chain over n instances of this grid size and
  // precision (ctx, phi, uhat: arrays of n), one launch per pass for all of
  // them (field_id() = instance). Each instance keeps its own fields, scratch,
  // model, symbol factors, flow words and step records; the partial sums,
  // tickets and scalars use one slot per instance in ctx[0]'s buffers, and
  // ctx[0]'s stream and tuning serve the launches. A stopped instance's blocks
  // return at once. The per-instance arithmetic does not depend on n.
  struct Step {
    spm_ctx *const *ctx;
    void *const *phi;
    void *const *uhat;
    int n;
    KParams base() const {
      KParams p = spm_params(ctx[0]);
      p.flow = ctx[0]->flow;
      p.stats = ctx[0]->stats;
      p.batched = n > 1;
      for (int b = 0; b < n; b++) {
        p.in[b] = p.out[b] = spm_buf(ctx[b], 0);
        if (n == 1) break;
        p.mb[b] = ctx[b]->m;
        p.gtabs[b] = reinterpret_cast<const double2 *>(ctx[b]->gtab);
        p.flows[b] = ctx[b]->flow;
        p.statss[b] = ctx[b]->stats;
      }
      return p;
    }
    int head() const {
      KParams p = base();
      for (int b = 0; b < n; b++) p.in[b] = phi[b];
      return plane_fwd<N, T, ProGrad<T>>(ctx[0], p, n);
    }
    // tiled_in / tiled_out: the spectrum u is read / written in tile order (the
    // chain's own copy) instead of the caller's array
    int spectral(bool tiled_in, bool tiled_out) const {
      KParams q = base();
      q.st_tiled = tiled_in;
      q.sto_tiled = tiled_out;
      for (int b = 0; b < n; b++) {
        q.st[b] = tiled_in ? spm_buf(ctx[b], 1) : uhat[b];
        q.sto[b] = tiled_out ? spm_buf(ctx[b], 1) : uhat[b];
      }
      return pencil<N, T, OpGrad<T>>(ctx[0], q, n);
    }
    // inverse -> forward; on a stopping step it stores phi and puts the tiled u
    // back into the caller's array
    int joint() const {
      KParams r = base();
      for (int b = 0; b < n; b++) {
        r.sto[b] = phi[b];
        r.aux0[b] = spm_buf(ctx[b], 1);
        r.aux1[b] = uhat[b];
      }
      return plane_inv_fwd<N, T, EpiFlow<T>, ProGrad<T>>(ctx[0], r, n);
    }
    int tail() const {
      KParams r = base();
      for (int b = 0; b < n; b++) r.out[b] = phi[b];
      return plane_inv<N, T, EpiFlow<T>>(ctx[0], r, n);
    }
  };

  // K gated steps as one chain: plane_fwd, then per step a pencil pass and the
  // joint inverse -> forward plane pass (the last step ends with plane_inv), so
  // phi crosses memory once per chain, and u stays in tile order between the
  // chain's first and last pencil pass.
  // With ev non-null (2K + 2 events) the chain records ev[0] before the head,
  // ev[1] after it and ev[2 + 2k], ev[3 + 2k] after step k's pencil and plane
  // pass (for per-kernel timing).
  static int chain(const Step &s, int K, void *const *ev) {
    auto rec = [&](int i) {
      if (ev) cudaEventRecord((cudaEvent_t)ev[i], s.ctx[0]->stream);
    };
    const bool fuse = s.ctx[0]->fuse_planes != 0;
    rec(0);
    SPM_TRY(s.head());
    rec(1);
    for (int k = 0; k < K; k++) {
      const bool last = k + 1 == K;
      SPM_TRY(s.spectral(fuse && k > 0, fuse && !last));
      rec(2 + 2 * k);
      if (last || !fuse) SPM_TRY(s.tail());
      else SPM_TRY(s.joint());
      rec(3 + 2 * k);
      if (!last && !fuse) SPM_TRY(s.head());
    }
    return 0;
  }
  static int grad_steps_ev(spm_ctx *c, void *phi, void *uhat, int K, void *const *ev) {
    SPM_NEED_SCRATCH(c, 2);
    return K <= 0 ? 0 : chain(Step{&c, &phi, &uhat, 1}, K, ev);
  }
  static int grad_steps(spm_ctx *c, void *phi, void *uhat, int K) { return grad_steps_ev(c, phi, uhat, K, nullptr); }
  static int grad_steps_group(spm_ctx *const *ctx, void *const *phi, void *const *uhat, int n, int K) {
    if (n < 1 || n > kMaxBatch) return spm_fail(SPM_ERR_ARG, "a group holds 1 to 16 instances");
    for (int b = 0; b < n; b++) {
      if (ctx[b]->N != N || ctx[b]->prec != ctx[0]->prec) return spm_fail(SPM_ERR_ARG, "a group shares N and precision");
      SPM_NEED_SCRATCH(ctx[b], 2);
    }
    return K <= 0 ? 0 : chain(Step{ctx, phi, uhat, n}, K, nullptr);
  }

  // -grad F(phi) -> grad, ||grad||^2 -> scal[SC_GN2]
  static int ngrad(spm_ctx *c, const void *phi, void *grad) {
    SPM_NEED_SCRATCH(c, 1);
    KParams p = spm_params(c);
    p.in[0] = phi;
    p.out[0] = spm_buf(c, 0);
    SPM_TRY((plane_fwd<N, T, ProNgrad<T>>(c, p, 1)));
    KParams q = spm_params(c);
    q.in[0] = spm_buf(c, 0);
    q.out[0] = spm_buf(c, 0);
    SPM_TRY((pencil<N, T, OpGmul<T, true>>(c, q, 1)));
    KParams r = spm_params(c);
    r.in[0] = spm_buf(c, 0);
    r.aux0[0] = phi;
    r.out[0] = grad;
    return plane_inv<N, T, EpiNgrad<T>>(c, r, 1);
  }

  // n <= kMaxBatch Hessian-vector products sharing phi.
  static int hv(spm_ctx *c, const void *phi, const void *const *v, void *const *hv, int n) {
    SPM_NEED_SCRATCH(c, n);
    KParams p = spm_params(c), q = spm_params(c), r = spm_params(c);
    for (int b = 0; b < n; b++) {
      p.in[b] = v[b];
      p.aux0[b] = phi;
      p.out[b] = spm_buf(c, b);
      q.in[b] = spm_buf(c, b);
      q.out[b] = spm_buf(c, b);
      r.in[b] = spm_buf(c, b);
      r.aux0[b] = phi;
      r.aux1[b] = v[b];
      r.out[b] = hv[b];
    }
    SPM_TRY((plane_fwd<N, T, ProHv<T>>(c, p, n)));
    SPM_TRY((pencil<N, T, OpGmul<T, false>>(c, q, n)));
    return plane_inv<N, T, EpiHv<T>>(c, r, n);
  }

  // n <= kMaxBatch Hessian products without their mean removal (EpiHvRaw):
  // v is transformed as it is, so phi is read once, by the epilogue.
  static int hv_raw(spm_ctx *c, const void *phi, const void *const *v, void *const *hv, int n) {
    SPM_NEED_SCRATCH(c, n);
    KParams p = spm_params(c), q = spm_params(c), r = spm_params(c);
    for (int b = 0; b < n; b++) {
      p.in[b] = v[b];
      p.out[b] = spm_buf(c, b);
      q.in[b] = spm_buf(c, b);
      q.out[b] = spm_buf(c, b);
      r.in[b] = spm_buf(c, b);
      r.aux0[b] = phi;
      r.aux1[b] = v[b];
      r.out[b] = hv[b];
    }
    SPM_TRY((plane_fwd<N, T, ProIdent<T>>(c, p, n)));
    SPM_TRY((pencil<N, T, OpGmul<T, false>>(c, q, n)));
    return plane_inv<N, T, EpiHvRaw<T>>(c, r, n);
  }

  // n <= kMaxBatch preconditioner applications, in place.
  static int precond(spm_ctx *c, void *const *w, int n) {
    SPM_NEED_SCRATCH(c, n);
    KParams p = spm_params(c), q = spm_params(c), r = spm_params(c);
    for (int b = 0; b < n; b++) {
      p.in[b] = w[b];
      p.out[b] = spm_buf(c, b);
      q.in[b] = spm_buf(c, b);
      q.out[b] = spm_buf(c, b);
      r.in[b] = spm_buf(c, b);
      r.out[b] = w[b];
    }
    SPM_TRY((plane_fwd<N, T, ProPrecond<T>>(c, p, n)));
    SPM_TRY((pencil<N, T, OpPrecond<T>>(c, q, n)));
    return plane_inv<N, T, EpiPrecond<T>>(c, r, n);
  }

  // <p, q> -> scal[SC_SUM0]
  static int dot(spm_ctx *c, const void *pp, const void *qq) {
    KParams p = spm_params(c);
    p.in[0] = pp;
    p.aux0[0] = qq;
    return reduce<N, T, ProDot<T>>(c, p, 1);
  }

  // Tangent preparation (get_Tv, SPM.cpp:15-32, plus what the force steps
  // need): with phi0 set, d = phi1 - phi0 is normalised and v = d/||d|| is
  // written to v_out; with phi0 null, phi1 is the tangent as given. Always
  // writes vhat = FFT(v)/N^3 (in tile order, state_index) and Gv = IFFT(G vhat, k = 0 removed).
  static int tangent(spm_ctx *c, const void *phi0, const void *phi1, void *v_out, void *vhat, void *gv) {
    SPM_NEED_SCRATCH(c, 1);
    KParams p = spm_params(c);
    p.in[0] = phi1;
    p.aux0[0] = phi0;
    p.out[0] = spm_buf(c, 0);
    SPM_TRY((plane_fwd<N, T, ProTangent<T>>(c, p, 1)));
    KParams q = spm_params(c);
    q.in[0] = spm_buf(c, 0);
    q.sto[0] = vhat;
    q.sto_tiled = 1;
    q.out[0] = spm_buf(c, 0);
    if (phi0) SPM_TRY((pencil<N, T, OpTangent<T, true>>(c, q, 1)));
    else SPM_TRY((pencil<N, T, OpTangent<T, false>>(c, q, 1)));
    KParams r = spm_params(c);
    r.in[0] = spm_buf(c, 0);
    r.aux0[0] = phi0;
    r.aux1[0] = phi1;
    r.sto[0] = phi0 ? v_out : nullptr;
    r.out[0] = gv;
    return plane_inv<N, T, EpiTangent<T>>(c, r, 1);
  }

  // Natural_Forces (factor 1) / MinMax_Forces (factor 2) on n fields in place,
  // all along the tangent (v, vhat, Gv) from tangent().
  static int force(spm_ctx *c, void *const *x, int n, const void *v, const void *vhat, const void *gv,
                   double factor) {
    SPM_NEED_SCRATCH(c, n);
    KParams p = spm_params(c), q = spm_params(c), r = spm_params(c);
    p.m.factor = factor;
    q.st_tiled = 1;
    for (int b = 0; b < n; b++) {
      p.in[b] = x[b];
      p.aux0[b] = v;
      p.aux1[b] = gv;
      p.out[b] = spm_buf(c, b);
      q.in[b] = spm_buf(c, b);
      q.st[b] = vhat;
      q.out[b] = spm_buf(c, b);
      r.in[b] = spm_buf(c, b);
      r.out[b] = x[b];
    }
    SPM_TRY((plane_fwd<N, T, ProForce<T>>(c, p, n)));
    SPM_TRY((pencil<N, T, OpForce<T>>(c, q, n)));
    return plane_inv<N, T, EpiStore<T>>(c, r, n);
  }

  // HiSD position step: x <- IFFT(Re(FFT(x + beta (N(x) - t)) / N^3 / (1 + beta G))), dx = x' - x.
  static int hisd_step(spm_ctx *c, void *x, const void *t, void *dx, double beta) {
    SPM_NEED_SCRATCH(c, 1);
    KParams p = spm_params(c);
    p.m.factor = beta;
    p.in[0] = x;
    p.aux0[0] = t;
    p.out[0] = spm_buf(c, 0);
    SPM_TRY((plane_fwd<N, T, ProHisd<T>>(c, p, 1)));
    KParams q = spm_params(c);
    q.m.factor = beta;
    q.in[0] = spm_buf(c, 0);
    q.out[0] = spm_buf(c, 0);
    SPM_TRY((pencil<N, T, OpHisd<T>>(c, q, 1)));
    KParams r = spm_params(c);
    r.in[0] = spm_buf(c, 0);
    r.aux1[0] = x;
    r.sto[0] = dx;
    r.out[0] = x;
    return plane_inv<N, T, EpiHisd<T>>(c, r, 1);
  }

  // ||ngrad(x_b)||^2 -> scal[b][SC_GN2] without storing the gradient.
  static int gnorm(spm_ctx *c, const void *const *x, int n) {
    SPM_NEED_SCRATCH(c, n);
    KParams p = spm_params(c), q = spm_params(c), r = spm_params(c);
    for (int b = 0; b < n; b++) {
      p.in[b] = x[b];
      p.out[b] = spm_buf(c, b);
      q.in[b] = spm_buf(c, b);
      q.out[b] = spm_buf(c, b);
      r.in[b] = spm_buf(c, b);
      r.aux0[b] = x[b];
      r.out[b] = nullptr;
    }
    SPM_TRY((plane_fwd<N, T, ProNgrad<T>>(c, p, n)));
    SPM_TRY((pencil<N, T, OpGmul<T, true>>(c, q, n)));
    return plane_inv<N, T, EpiNgrad<T>>(c, r, n);
  }

  static const OpsTable *table() {
    using X = std::conditional_t<sizeof(T) == 4, clu::Chains<N, float>, Impl>;
    static const OpsTable t = {&X::fft, &X::ifft, &X::energy, &X::grad_step, &X::grad_steps, &X::grad_steps_ev,
                               &X::grad_step_ev, &X::ngrad, &hv, &precond, &dot, &tangent, &force, &gnorm,
                               &hisd_step, &X::grad_steps_group, &hv_raw};
    return &t;
  }
};

}  // namespace spm
