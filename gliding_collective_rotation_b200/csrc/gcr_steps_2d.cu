// gcr_steps_2d.cu -- the one-kernel steps in 2D, FP64.
#include "gcr_phases.cuh"

namespace gcr {

void steps_kernels_2d(KernelSet &k)
{
    k.steps[0] = (void *)k_steps<2, double, 0>;
    k.steps[1] = (void *)k_steps<2, double, 1>;
    k.steps[2] = (void *)k_steps<2, double, 2>;
}

}  // namespace gcr
