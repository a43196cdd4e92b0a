// Two-step Λ pass, lengths of group 3 (splits.cuh).
#include "apply_lam.cuh"

namespace mrsr {
MRSR_LAMBDA_GROUP(3)
}  // namespace mrsr
