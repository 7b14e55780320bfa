// Instances of the day kernel: one variant, no curfew.
#include "psim_day.cuh"

namespace psim {

DayKernel day_kernel_a(int instance) {
    return instance == DAY_ONE_PLAIN ? k_day<1, false, 0> : k_day<1, false, 1>;
}

}  // namespace psim
