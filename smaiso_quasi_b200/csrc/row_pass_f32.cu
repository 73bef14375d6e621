// z passes in float.
#include "row_pass.cuh"

namespace quasi {
QUASI_INSTANTIATE_ROW_PASS(float)
}  // namespace quasi
