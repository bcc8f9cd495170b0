// period3.cu -- the period kernel in 3 dimensions.
#include "period_launch.cuh"

namespace rd {
template struct PeriodOf<3>;
}  // namespace rd
