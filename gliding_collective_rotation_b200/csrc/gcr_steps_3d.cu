// gcr_steps_3d.cu -- the one-kernel steps in 3D, FP64.
#include "gcr_phases.cuh"

namespace gcr {

void steps_kernels_3d(KernelSet &k)
{
    k.steps[0] = (void *)k_steps<3, double, 0>;
    k.steps[1] = (void *)k_steps<3, double, 1>;
    k.steps[2] = (void *)k_steps<3, double, 2>;
}

}  // namespace gcr
