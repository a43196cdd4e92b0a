// Two-step Λ pass, lengths of group 4 (splits.cuh).
#include "apply_lam.cuh"

namespace mrsr {
MRSR_LAMBDA_GROUP(4)
}  // namespace mrsr
