// Two-step row and middle passes, lengths of group 4 (splits.cuh).
#include "apply_fast.cuh"

namespace mrsr {
MRSR_ROWS_GROUP(4)
}  // namespace mrsr
