// Launch helpers shared by the kernel chains.
#pragma once

#include <atomic>
#include <type_traits>

#include "../../include/spmiqc.h"
#include "blas1.cuh"
#include "spm_internal.h"
#include "spm_table.h"

namespace spm {

#define SPM_TRY(x)               \
  do {                           \
    int _s = (x);                \
    if (_s != 0) return _s;      \
  } while (0)

// Every chain that goes through the spectral scratch checks that the caller
// made room for its fields (spm_ensure_scratch) instead of writing through an
// unallocated buffer.
#define SPM_NEED_SCRATCH(c, nf)                                                         \
  do {                                                                                  \
    if ((c)->scratch_cap < (nf) || !(c)->buf)                                           \
      return spm_fail(SPM_ERR_STATE, "spectral scratch not allocated for this batch"); \
  } while (0)

// Sets the dynamic shared-memory limit of a kernel once per device. Tag makes
// the "done" bits distinct per kernel (the kernels share one function type).
template <class Tag, class K> static cudaError_t prepare(K kern, size_t smem, int dev) {
  // one bit per device (first 32); contexts on several host threads may race
  // here, which at worst sets the attribute twice
  static std::atomic<unsigned> done{0};
  if (dev < 32 && (done.load(std::memory_order_acquire) >> dev) & 1u) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && dev < 32) done.fetch_or(1u << dev, std::memory_order_release);
  return e;
}

// Programmatic dependent launches (knob "pdl"); a stream capture turns them
// into programmatic edges of the graph.
static inline bool pdl_on(const spm_ctx *c) { return c->pdl != 0; }

template <int N, class T, class F> static int reduce(spm_ctx *c, const KParams &p, int nb) {
  constexpr size_t npairs = (size_t)N * N * N / 2;
  constexpr int blocks = (int)((npairs + kThreads - 1) / kThreads < (size_t)kReduceBlocks
                                   ? (npairs + kThreads - 1) / kThreads
                                   : (size_t)kReduceBlocks);
  c->launches++;
  field_reduce_kernel<T, F><<<dim3(blocks, nb, 1), kThreads, 0, c->stream>>>(p, npairs);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : spm_fail_cuda(e, "reduce launch");
}

}  // namespace spm
