// Autotuner for the transform schedule of a context (no counterpart in the
// reference; FFTW's plan search plays this role there, My_FFT.cpp:49-97).
// FP64 contexts (tile passes): whether gradient chains use the fused inverse ->
// forward plane pass, and programmatic dependent launches or not (knob "pdl").
// FP32 contexts (cluster passes): the plane-pass variant (staged with one CTA per SM, direct loads
// with two CTAs per SM, or three CTAs per SM with fewer registers per thread),
// the fused plane pass or not, and
// whether their plane kernels exchange through distributed shared memory or
// through global areas resident in L2; then, for the fastest, the pencil tile
// width and programmatic dependent launches (knob "pdl").
// Tuning an FP64 context also chooses the FP32 schedule of its twin (mixed flows).
// Each candidate runs a short chain of gradient steps on a scratch field with
// CUDA events around it; the fastest is kept in the context and remembered per
// (device, N, precision) for later contexts.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "../../include/spmiqc.h"
#include "spm_internal.h"

namespace {

std::mutex g_mu;
struct Choice {
  int plane_cps, fuse_planes, plane_xg, pencil_tc = 8, pdl = 0;
};
std::map<std::tuple<int, int, int>, Choice> g_best;  // (device, N, prec) -> schedule
std::map<std::tuple<int, int, int>, Choice> g_twin;  // the same for twins of tuned FP64 contexts

// A smooth non-trivial field (a few cosines), so the timed steps do real work
// and the flow does not stop on its first step.
template <class T> __global__ void fill_kernel(T *phi, int N) {
  const size_t n = (size_t)N * N * N;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i / ((size_t)N * N)), y = (int)((i / N) % N), z = (int)(i % N);
    phi[i] = (T)(0.1 * (cospi(2.0 * (3 * x + 5 * y) / N) + sinpi(2.0 * (7 * z - 2 * x) / N)) +
                 1e-3 * ((x * 31 + y * 17 + z * 13) % 29) / 29.0);
  }
}

// The knobs that concern the context's kernels: an FP64 one keeps those that
// only its FP32 twin reads.
void apply(spm_ctx *c, const Choice &ch) {
  c->fuse_planes = ch.fuse_planes;
  c->pdl = ch.pdl;
  if (c->prec == SPM_FP64) return;
  c->plane_cps = ch.plane_cps;
  c->plane_xg = ch.plane_xg;
  c->pencil_tc = ch.pencil_tc;
}

// Times the candidates on the context; leaves its knobs changed.
int search(spm_ctx *c, int steps, Choice *out) {
  void *phi = nullptr, *uh = nullptr;
  cudaError_t e = cudaMalloc(&phi, c->field_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&uh, c->field_bytes);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  int rc = e == cudaSuccess ? SPM_OK : spm_fail_cuda(e, "autotune buffers");
  Choice best = {c->plane_cps, c->fuse_planes, c->plane_xg, c->pencil_tc, c->pdl};
  float best_ms = 1e30f;
  // plane variant, fused plane pass, exchange routes of the gradient chains
  const Choice cands[] = {{2, 1, 0}, {3, 1, 0}, {1, 1, 0}, {2, 0, 0}, {2, 1, spm::kXgFwd | spm::kXgInv},
                          {3, 1, spm::kXgFwd | spm::kXgInv}, {2, 1, spm::kXgFwd}, {2, 1, spm::kXgInv}};
  std::vector<Choice> all(std::begin(cands), std::end(cands));
  // FP64 chains run on the tile passes, without variants of the planes (the list
  // does not depend on the context: the choice serves later ones too)
  if (c->prec == SPM_FP64) all = {{2, 1, 0}, {2, 0, 0}};
  if (c->prec == SPM_FP32) all.push_back({4, 1, spm::kXgFwd | spm::kXgInv});  // four CTAs per SM
  if (c->prec == SPM_FP32) {
    all.push_back({5, 1, spm::kXgFwd | spm::kXgInv});  // 16-row CTAs, four per SM
    all.push_back({6, 1, spm::kXgFwd | spm::kXgInv});  // the same, fused pass pipelined over planes
  }
  // best of three timed chains of `steps` gated steps with the candidate's knobs
  auto time_it = [&](const Choice &cand, float &t) -> int {
    apply(c, cand);
    int r = spm_ensure_xg(c);
    if (r != SPM_OK) return r;
    if (c->prec == SPM_FP64) fill_kernel<double><<<592, 256, 0, c->stream>>>((double *)phi, c->N);
    else fill_kernel<float><<<592, 256, 0, c->stream>>>((float *)phi, c->N);
    r = spm_fft(c, phi, uh);
    // warm-up (kernel attributes, occupancy queries, caches), then the best of three timed chains
    if (r == SPM_OK) r = spm_grad_flow_enqueue(c, phi, uh, 3, 0.0);
    if (r == SPM_OK) r = spm_grad_flow_collect(c, nullptr, 0, nullptr);
    t = 1e30f;
    for (int rep = 0; rep < 3 && r == SPM_OK; rep++) {
      cudaEventRecord(e0, c->stream);
      r = spm_grad_flow_enqueue(c, phi, uh, steps, 0.0);
      cudaEventRecord(e1, c->stream);
      if (r == SPM_OK) r = spm_grad_flow_collect(c, nullptr, 0, nullptr);
      float ms = 0;
      if (r == SPM_OK && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess && ms < t) t = ms;
    }
    return r;
  };
  for (const Choice &cand : all) {
    if (rc != SPM_OK) break;
    float t = 1e30f;
    rc = time_it(cand, t);
    // a later candidate must be at least 1 % faster to replace the best so far
    // (candidates within timing noise of each other resolve to the earlier one)
    if (rc == SPM_OK && t < 0.99f * best_ms) {
      best_ms = t;
      best = cand;
    }
  }
  // then the pencil tile width for the best schedule: 4-column tiles (several
  // CTAs per SM) if they are at least 1 % faster
  if (rc == SPM_OK && c->prec == SPM_FP32) {
    Choice narrow = best;
    narrow.pencil_tc = 4;
    float t = 1e30f;
    rc = time_it(narrow, t);
    if (rc == SPM_OK && t < 0.99f * best_ms) {
      best_ms = t;
      best = narrow;
    }
  }
  // and programmatic dependent launches of the plane and pencil kernels, if
  // they are at least 1 % faster
  if (rc == SPM_OK) {
    Choice dep = best;
    dep.pdl = 1;
    float t = 1e30f;
    rc = time_it(dep, t);
    if (rc == SPM_OK && t < 0.99f * best_ms) {
      best_ms = t;
      best = dep;
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(phi);
  cudaFree(uh);
  if (rc == SPM_OK) *out = best;
  return rc;
}

// The schedule of an FP64 context's FP32 twin: what an FP32 context of the size
// has been tuned to, else the fastest on a context made for the search. Without
// room for that one the twin keeps the FP64 context's knobs.
void tune_twin(spm_ctx *c, int steps) {
  const auto key = std::make_tuple(c->device, c->N, (int)SPM_FP32);
  Choice ch;
  bool known = false;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto *m : {&g_best, &g_twin}) {
      auto it = m->find(key);
      if (known || it == m->end()) continue;
      ch = it->second;
      known = true;
    }
  }
  if (!known) {
    spm_ctx *t = nullptr;
    int rc = spm_ctx_create(c->N, c->L, c->m.Tau, c->m.Gamma, c->m.dt, SPM_FP32, c->stream, &t);
    if (rc == SPM_OK) rc = search(t, steps, &ch);
    if (t) spm_ctx_destroy(t);
    if (rc != SPM_OK) {
      cudaGetLastError();  // a refused allocation
      return;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    g_twin[key] = ch;
  }
  c->twin_plane_cps = ch.plane_cps;
  c->twin_fuse_planes = ch.fuse_planes;
  c->twin_plane_xg = ch.plane_xg;
  c->twin_pencil_tc = ch.pencil_tc;
  c->twin_pdl = ch.pdl;
  c->twin_tuned = true;
}

}  // namespace

// The remembered choice for (device, N, precision), if any.
bool spm_autotune_lookup(int device, int N, int prec, int *plane_cps, int *fuse_planes, int *plane_xg,
                         int *pencil_tc, int *pdl) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_best.find(std::make_tuple(device, N, prec));
  if (it == g_best.end()) return false;
  *plane_cps = it->second.plane_cps;
  *fuse_planes = it->second.fuse_planes;
  *plane_xg = it->second.plane_xg;
  if (pencil_tc) *pencil_tc = it->second.pencil_tc;
  if (pdl) *pdl = it->second.pdl;
  return true;
}

extern "C" int spm_autotune(spm_ctx *c, int steps, int *plane_cps, int *fuse_planes) {
  if (!c || steps < 2) return spm_fail(SPM_ERR_ARG, "bad argument (steps >= 2)");
  const auto key = std::make_tuple(c->device, c->N, c->prec);
  auto finish = [&](const Choice &ch) {
    apply(c, ch);
    if (!c->plane_xg && c->xg) {  // the exchange areas are not used by the chosen schedule
      cudaStreamSynchronize(c->stream);
      cudaFree(c->xg);
      c->xg = nullptr;
      c->xg_cap = 0;
    }
    if (plane_cps) *plane_cps = c->plane_cps;
    if (fuse_planes) *fuse_planes = c->fuse_planes;
    return spm_ensure_xg(c);
  };
  Choice ch;
  bool known = false;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_best.find(key);
    if (it != g_best.end()) {
      ch = it->second;
      known = true;
    } else if (auto tw = g_twin.find(key); tw != g_twin.end()) {  // (FP32) searched for a twin before
      ch = g_best[key] = tw->second;
      known = true;
    }
  }
  if (!known) {
    const Choice saved = {c->plane_cps, c->fuse_planes, c->plane_xg, c->pencil_tc, c->pdl};
    const int rc = search(c, steps, &ch);
    if (rc != SPM_OK) {
      finish(saved);
      return rc;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    g_best[key] = ch;
  }
  const int rc = finish(ch);
  if (rc == SPM_OK && c->prec == SPM_FP64) tune_twin(c, steps);
  return rc;
}
