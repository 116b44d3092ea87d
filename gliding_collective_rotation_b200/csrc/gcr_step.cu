// gcr_step.cu -- the kernels of the launch-by-launch step, and the table of
// all step kernels of a dimension and precision.
#include "gcr_phases.cuh"

namespace gcr {

// one CTA: the per-system work between two kernels of a step
__global__ void __launch_bounds__(1024) k_duty(const __grid_constant__ BatchArgs A, int duty)
{
    pdl_wait();
    if (duty == kDutyDt) {
        for (int i = threadIdx.x; i < A.n_slots; i += blockDim.x) sys_dt(A, i);
        return;
    }
    step_duty(A, duty);
}

// ... of many systems: a thread a slot, and the last CTA to finish makes the plan
// (4096 systems of 30 beads 183 us a step with one CTA, 130 so; 16,384 of 10 522
// and 276).  A kernel of its own: with this in k_duty a step of few systems, whose
// launches begin with cold instruction caches, took 0.8 us more.
__global__ void __launch_bounds__(1024) k_duty_wide(const __grid_constant__ BatchArgs A, int duty)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (duty == kDutyDt) {
        if (i < A.n_slots) sys_dt(A, i);
        return;
    }
    const int used = *A.n_used;
    const unsigned ctas = max(1, (used + (int)blockDim.x - 1) / (int)blockDim.x);
    if (blockIdx.x >= ctas) return;
    if (duty == kDutyEnd && i < used) sys_end(A, i);
    const int ask = __syncthreads_or(i < used && asks_build(A.P[i], A.S[i]));
    __threadfence();
    __syncthreads();
    unsigned done = 0;
    if (threadIdx.x == 0) done = atomicAdd(A.duty_done, 1u + (ask ? 65536u : 0u)) + 1u + (ask ? 65536u : 0u);
    if (!__syncthreads_or((done & 65535u) == ctas)) return;
    if (threadIdx.x == 0) *A.duty_done = 0;
    __threadfence();
    make_plan(A, __syncthreads_or(done >> 16));
}

__global__ void __launch_bounds__(512) k_sort(const __grid_constant__ BatchArgs A)
{
    pdl_wait();
    sort_tiles(A, list_span());
}

// chain-neighbour bits of every bead of one system
__global__ void k_topo(const int32_t *__restrict__ chain, int n, uint8_t *topo)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    int c = chain[b];
    uint8_t t = 0;
    if (b >= 1 && chain[b - 1] == c) t |= kHasPrev;
    if (b >= 2 && chain[b - 2] == c) t |= kHasPrev2;
    if (b + 1 < n && chain[b + 1] == c) t |= kHasNext;
    if (b + 2 < n && chain[b + 2] == c) t |= kHasNext2;
    topo[b] = t;
}

// flag system `slot` for a list build (every resident system when slot < 0):
// admission, a new descriptor, a coupling change
__global__ void k_sys_mark(BatchArgs A, int n_slots, int slot)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_slots || (slot >= 0 && i != slot)) return;
    A.S[i].rebuild = 1;
}

// ------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------
template <int D, typename FT>
struct StepKernels {
    static void *pair0() { return (void *)k_pair<D, FT, 0, false>; }
    static void *pair1() { return (void *)k_pair<D, FT, 1, false>; }
    static void *pair_cells0() { return (void *)k_pair_cells<D, FT, 0>; }
    static void *pair_cells1() { return (void *)k_pair_cells<D, FT, 1>; }
    static void *update() { return (void *)k_update<D, FT>; }
    static void *rigid0() { return (void *)k_rigid<D, FT, 0>; }
    static void *rigid1() { return (void *)k_rigid<D, FT, 1>; }
    // stages 0, 1 and 10..13 (SRK4), with the pair forces of k_pair or their own
    static void fill_stages(KernelSet &k)
    {
        k.stage[0] = (void *)k_stage<D, FT, 0>;
        k.stage[1] = (void *)k_stage<D, FT, 1>;
        k.stage_own[0] = (void *)k_stage<D, FT, 0, true>;
        k.stage_own[1] = (void *)k_stage<D, FT, 1, true>;
        // SRK4: with their own in 2D mixed precision, else (and coupled) k_pair's
        k.stage[2] = (void *)k_stage<D, FT, 10>;
        k.stage[3] = (void *)k_stage<D, FT, 11>;
        k.stage[4] = (void *)k_stage<D, FT, 12>;
        k.stage[5] = (void *)k_stage<D, FT, 13>;
        if constexpr (D == 2 && sizeof(FT) == 4) {
            k.stage_own[2] = (void *)k_stage<D, FT, 10, true>;
            k.stage_own[3] = (void *)k_stage<D, FT, 11, true>;
            k.stage_own[4] = (void *)k_stage<D, FT, 12, true>;
            k.stage_own[5] = (void *)k_stage<D, FT, 13, true>;
        }
    }
    static void fill4(KernelSet &k)
    {
        k.pair2 = (void *)k_pair<D, FT, 2, false>;
        k.rigid4[0] = (void *)k_rigid<D, FT, 10>;
        k.rigid4[1] = (void *)k_rigid<D, FT, 11>;
        k.rigid4[2] = (void *)k_rigid<D, FT, 12>;
        k.rigid4[3] = (void *)k_rigid<D, FT, 13>;
        k.pair_cross[0] = (void *)k_pair<D, FT, 0, true>;
        k.pair_cross[1] = (void *)k_pair<D, FT, 1, true>;
        k.pair_cross[2] = (void *)k_pair<D, FT, 2, true>;
    }
};

KernelSet kernel_set(int dim, int precision)
{
    KernelSet k{};
    if (dim == 2)
        precision == 0 ? steps_kernels_2d(k) : steps_kernels_2f(k);
    else
        precision == 0 ? steps_kernels_3d(k) : steps_kernels_3f(k);
    if (dim == 2)
        k.pair_smem = precision == 0 ? pair_smem_bytes<2, double> : pair_smem_bytes<2, float>;
    else
        k.pair_smem = precision == 0 ? pair_smem_bytes<3, double> : pair_smem_bytes<3, float>;
    k.pair_cells_smem = dim == 2 ? pair_cells_smem_bytes<2> : pair_cells_smem_bytes<3>;
    k.pair_cells_rows = dim == 2 ? 3 : 9;
    k.max_row_cells = kMaxRowCells;
#define GCR_FILL(D_, FT_)                       \
    k.pair0 = StepKernels<D_, FT_>::pair0();    \
    k.pair1 = StepKernels<D_, FT_>::pair1();    \
    k.pair_cells[0] = StepKernels<D_, FT_>::pair_cells0(); \
    k.pair_cells[1] = StepKernels<D_, FT_>::pair_cells1(); \
    k.update = StepKernels<D_, FT_>::update();  \
    k.rigid0 = StepKernels<D_, FT_>::rigid0();  \
    k.rigid1 = StepKernels<D_, FT_>::rigid1();  \
    StepKernels<D_, FT_>::fill_stages(k);        \
    StepKernels<D_, FT_>::fill4(k);
    if (dim == 2 && precision == 0) {
        GCR_FILL(2, double)
    } else if (dim == 2) {
        GCR_FILL(2, float)
    } else if (precision == 0) {
        GCR_FILL(3, double)
    } else {
        GCR_FILL(3, float)
    }
#undef GCR_FILL
    if (dim == 2) {
        k.bin0 = (void *)k_bin<2, 0>;
        k.bin1 = (void *)k_bin<2, 1>;
        k.build0 = (void *)k_build<2, 0>;
        k.build1 = (void *)k_build<2, 1>;
        k.bin2 = (void *)k_bin<2, 2>;
        k.build2 = (void *)k_build<2, 2>;
        k.run_check = (void *)k_run_check<2>;
        k.motor[0] = (void *)k_motor<2, 0>;
        k.motor[1] = (void *)k_motor<2, 1>;
    } else {
        k.bin0 = (void *)k_bin<3, 0>;
        k.bin1 = (void *)k_bin<3, 1>;
        k.build0 = (void *)k_build<3, 0>;
        k.build1 = (void *)k_build<3, 1>;
        k.bin2 = (void *)k_bin<3, 2>;
        k.build2 = (void *)k_build<3, 2>;
        k.run_check = (void *)k_run_check<3>;
        k.motor[0] = (void *)k_motor<3, 0>;
        k.motor[1] = (void *)k_motor<3, 1>;
    }
    k.sort = (void *)k_sort;
    k.topo = (void *)k_topo;
    k.sys_mark = (void *)k_sys_mark;
    k.duty = (void *)k_duty;
    k.duty_wide = (void *)k_duty_wide;
    return k;
}

}  // namespace gcr
