// Two-step Λ pass, lengths of group 5 (splits.cuh).
#include "apply_lam.cuh"

namespace mrsr {
MRSR_LAMBDA_GROUP(5)
}  // namespace mrsr
