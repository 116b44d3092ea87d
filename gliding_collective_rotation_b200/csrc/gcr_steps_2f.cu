// gcr_steps_2f.cu -- the one-kernel steps in 2D, mixed precision.
#include "gcr_phases.cuh"

namespace gcr {

void steps_kernels_2f(KernelSet &k)
{
    k.steps[0] = (void *)k_steps<2, float, 0>;
    k.steps[1] = (void *)k_steps<2, float, 1>;
    k.steps[2] = (void *)k_steps<2, float, 2>;
}

}  // namespace gcr
