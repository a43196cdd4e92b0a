// Two-step row and middle passes, lengths of group 5 (splits.cuh).
#include "apply_fast.cuh"

namespace mrsr {
MRSR_ROWS_GROUP(5)
}  // namespace mrsr
