// Two-step row and middle passes, lengths of groups 1 and 2 (splits.cuh).
#include "apply_fast.cuh"

namespace mrsr {
MRSR_ROWS_GROUP(1)
MRSR_ROWS_GROUP(2)
}  // namespace mrsr
