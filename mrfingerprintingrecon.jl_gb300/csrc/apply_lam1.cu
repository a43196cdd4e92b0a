// Two-step Λ pass, lengths of group 1 (splits.cuh).
#include "apply_lam.cuh"

namespace mrsr {
MRSR_LAMBDA_GROUP(1)
}  // namespace mrsr
