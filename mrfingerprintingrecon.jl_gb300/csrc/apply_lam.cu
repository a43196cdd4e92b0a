// Two-step Λ pass (apply_lam.cuh): dispatch over the compiled lengths, and their first group.
#include "apply_lam.cuh"

namespace mrsr {

MRSR_LAMBDA_GROUP(0)

int fast_lambda(const LamPassArgs& a, int ncg, cudaStream_t st) {
  for (auto* f : {lambda_group_0, lambda_group_1, lambda_group_2, lambda_group_3, lambda_group_4, lambda_group_5}) {
    const int s = f(a, ncg, st);
    if (s != MRSR_ERR_UNSUPPORTED) return s;
  }
  return MRSR_ERR_UNSUPPORTED;
}

}  // namespace mrsr
