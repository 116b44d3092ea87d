// gcr_steps_3f.cu -- the one-kernel steps in 3D, mixed precision.
#include "gcr_phases.cuh"

namespace gcr {

void steps_kernels_3f(KernelSet &k)
{
    k.steps[0] = (void *)k_steps<3, float, 0>;
    k.steps[1] = (void *)k_steps<3, float, 1>;
    k.steps[2] = (void *)k_steps<3, float, 2>;
}

}  // namespace gcr
