// z passes in double.
#include "row_pass.cuh"

namespace quasi {
QUASI_INSTANTIATE_ROW_PASS(double)
}  // namespace quasi
