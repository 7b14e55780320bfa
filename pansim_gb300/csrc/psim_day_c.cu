// Instances of the day kernel: two variants without a curfew, any context.
#include "psim_day.cuh"

namespace psim {

DayKernel day_kernel_c(int instance) {
    return instance == DAY_TWO ? k_day<2, false, 1> : k_day<0, true, 2>;
}

}  // namespace psim
