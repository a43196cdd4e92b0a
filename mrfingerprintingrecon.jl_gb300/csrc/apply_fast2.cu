// Two-step row and middle passes, lengths of group 3 (splits.cuh).
#include "apply_fast.cuh"

namespace mrsr {
MRSR_ROWS_GROUP(3)
}  // namespace mrsr
