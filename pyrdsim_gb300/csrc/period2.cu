// period2.cu -- the period kernel in 2 dimensions.
#include "period_launch.cuh"

namespace rd {
template struct PeriodOf<2>;
}  // namespace rd
