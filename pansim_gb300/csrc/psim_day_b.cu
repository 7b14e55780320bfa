// Instances of the day kernel: one variant with a curfew, one variant with
// expected infections or the adjoint.
#include "psim_day.cuh"

namespace psim {

DayKernel day_kernel_b(int instance) {
    return instance == DAY_ONE_CURFEW ? k_day<1, false, 2> : k_day<1, true, 0>;
}

}  // namespace psim
