// Instances of the day kernel: one variant, no curfew, the grid one cluster.
#include "psim_day.cuh"

namespace psim {

DayKernel day_kernel_d(int instance) {
    return instance == DAY_ONE_PLAIN_CLUSTER ? k_day<1, false, 0, true> : k_day<1, false, 1, true>;
}

}  // namespace psim
