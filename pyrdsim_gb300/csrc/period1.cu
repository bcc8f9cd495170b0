// period1.cu -- the period kernel in 1 dimension.
#include "period_launch.cuh"

namespace rd {
template struct PeriodOf<1>;
}  // namespace rd
