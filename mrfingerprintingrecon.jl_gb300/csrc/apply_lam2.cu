// Two-step Λ pass, lengths of group 2 (splits.cuh).
#include "apply_lam.cuh"

namespace mrsr {
MRSR_LAMBDA_GROUP(2)
}  // namespace mrsr
