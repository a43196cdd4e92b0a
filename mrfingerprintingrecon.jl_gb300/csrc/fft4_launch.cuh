// Launch helpers of the register two-step kernels (apply_fast.cuh, apply_lam.cuh).
#pragma once
#include "fft4.cuh"
#include "passes.cuh"
#include "splits.cuh"

namespace mrsr {

inline Slots make_slots(int R2, int TC) {
  Slots s;
  s.TC = TC;
  s.tcs = 0;
  while ((1 << s.tcs) < TC) ++s.tcs;
  s.W = slots_width(R2, TC);
  return s;
}

template <class K, class A, class SL>
int launch(K k, dim3 grid, int threads, size_t smem, cudaStream_t st, const A& a, const SL& sl) {
  MRSR_REQUIRE(smem <= 227 * 1024, MRSR_ERR_UNSUPPORTED, "shared memory request %zu too large", smem);
  if (smem > 48 * 1024) MRSR_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  MRSR_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  return launch_dependent(k, grid, threads, smem, st, a, sl);
}

}  // namespace mrsr
