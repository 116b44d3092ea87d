// gcr_observables.cu -- the reference's analysis observables on the device.
//
// Chain frames (analysis.chain_COM, analysis.py:288-292; the mean chain angle
// output_methods.calc_avg_phi_chain, output_methods.py:492-510) and the pair
// correlations over chain centres (analysis.correlation_func with g_of_r,
// Cvv, Cnn, analysis.py:203-275), for the resident systems of a context.
// The reference computes them in Python loops, O(n_chains^2) for the
// correlations; here one thread per chain, and for the pairs a thread per row
// of a tile of 64 x 64 chains (or of a slice of its columns).
//
// Determinism: g(r) counts are integers; the Cvv / Cnn sums are accumulated
// in 64-bit fixed point (2^-32 resolution per pair), so the histograms do not
// depend on the order of the atomic additions.  Separations use explicitly
// rounded products and sums, as numpy evaluates them.
#include "gcr_device.cuh"
#include "gcr_kernels.h"

namespace gcr {

// analysis.true_sep (analysis.py:185-187): np.mod(pt2 - pt1 + L/2, L) - L/2
__device__ __forceinline__ double true_sep(double pt1, double pt2, double L)
{
    return __dsub_rn(py_mod(__dadd_rn(__dsub_rn(pt2, pt1), 0.5 * L), L), 0.5 * L);
}

// one thread per chain: the reference's chain "centre" (head + sum of the
// separations head - x_i, wrapped: analysis.chain_COM as written) and the
// mean angle of the tangents with 1- and 2-fold symmetry; trig (sym 1 or 2):
// cosine and sine of that angle, for the pair sums
template <int D, typename FT>
__global__ void k_chain_frame(const double *__restrict__ pos, const FT *__restrict__ tan,
                              const int32_t *__restrict__ cs, int n_chains, double L, double *com, double *phi,
                              int sym, double *trig)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_chains) return;
    const int b0 = cs[c], b1 = cs[c + 1];
    if (com) {
        double head[D], acc[D];
#pragma unroll
        for (int i = 0; i < D; i++) {
            head[i] = pos[(size_t)b0 * D + i];
            acc[i] = 0.0;
        }
#pragma unroll 4
        for (int b = b0; b < b1; b++)
#pragma unroll
            for (int i = 0; i < D; i++) acc[i] = __dadd_rn(acc[i], true_sep(pos[(size_t)b * D + i], head[i], L));
#pragma unroll
        for (int i = 0; i < D; i++) com[(size_t)c * D + i] = py_mod(__dadd_rn(head[i], acc[i]), L);
    }
    if (!phi && !trig) return;
    double sx = 0.0, sy = 0.0, s2 = 0.0, c2 = 0.0;
#pragma unroll 2
    for (int b = b0; b < b1; b++) {
        const double tx = (double)tan[(size_t)b * D], ty = (double)tan[(size_t)b * D + 1];
        sx = __dadd_rn(sx, tx);
        sy = __dadd_rn(sy, ty);
        if (!phi && sym == 1) continue;
        const double a = atan2(ty, tx);
        double sn, cn;
        sincos(2.0 * a, &sn, &cn);
        s2 = __dadd_rn(s2, sn);
        c2 = __dadd_rn(c2, cn);
    }
    if (phi) {
        phi[(size_t)c * 2] = atan2(sy, sx);
        phi[(size_t)c * 2 + 1] = atan2(s2, c2) / 2.0;
    }
    if (trig) {
        const double a = sym == 1 ? atan2(sy, sx) : atan2(s2, c2) / 2.0;
        trig[(size_t)c * 2] = cos(a);
        trig[(size_t)c * 2 + 1] = sin(a);
    }
}

constexpr double kFix = 4294967296.0;  // 2^32: fixed-point scale of the pair sums

// true_sep of two centres, which lie in [0, L): one wrap at most
__device__ __forceinline__ double centre_sep(double pt1, double pt2, double L)
{
    const double x = __dadd_rn(__dsub_rn(pt2, pt1), 0.5 * L);
    if (!(x > -L && x < 2.0 * L)) return __dsub_rn(py_mod(x, L), 0.5 * L);
    return __dsub_rn(x < 0.0 ? __dadd_rn(x, L) : (x >= L ? __dsub_rn(x, L) : x), 0.5 * L);
}

// the reference's bin of a squared distance, int(sqrt(d2) / binsize).  In FP32
// first: its quotient is within 3e-7 of the exact one, relative, so unless it
// lies that near a bin's edge the bin is decided; else the exact FP64 square
// root and division, about 60 instructions, decide.
__device__ __forceinline__ long long pair_bin(double d2, double binsize, float inv)
{
    const float q = sqrtf((float)d2) * inv;
    const float f = floorf(q), edge = 1e-6f * q + 1e-5f;
    if (q - f > edge && f + 1.0f - q > edge && q < 1e6f) return (long long)f;
    return (long long)__ddiv_rn(sqrt(d2), binsize);
}

// Chain pairs (i > j), tiles of kPairTile x kPairTile chains, kPairGroups of
// them a CTA at a time: a thread a row of its tile, the columns in shared
// memory, one histogram a CTA.  Bound by FP64 issue and, with few chains, by
// launches.  One pair a thread, with its row found by a square root, a sine
// and a cosine of both angles for every pair and three allocations a call took
// 185 us a call for g(r) and 265 us for Cvv and Cnn of 4000 chains; so 85 and
// 102 us (B200, host to host; the kernel 38 and 52 us).  While there are fewer
// tiles than groups on the SMs, a tile's columns are cut into up to kPairSlices
// slices, a group each: a thread that walks all 64 alone is the time of a call
// with few chains (the five calls of an analysis of 50, 500 and 1400 chains 355,
// 392 and 397 us with whole tiles, 288, 307 and 348 so).
constexpr int kPairTile = 64, kPairGroups = 4, kPairSlices = 16;

__global__ void __launch_bounds__(kPairTile *kPairGroups)
    k_pair_corr(const double *__restrict__ com, const double *__restrict__ trig, int n_chains, double L, double binsize,
                int n_bins, int kind, int slices, unsigned long long *counts, unsigned long long *sums)
{
    extern __shared__ unsigned long long sh_hist[];  // kinds 1, 2: [n_bins] fixed-point sums; [n_bins] 32-bit counts
    unsigned long long *hs = sh_hist;
    unsigned *hc = reinterpret_cast<unsigned *>(sh_hist + (kind != 0 ? n_bins : 0));
    __shared__ double col[kPairGroups][4][kPairTile];  // x, y, cosine, sine
    for (int i = threadIdx.x; i < n_bins; i += blockDim.x) {
        hc[i] = 0u;
        if (kind != 0) hs[i] = 0ull;
    }
    const int group = threadIdx.x / kPairTile, lane = threadIdx.x % kPairTile;
    const double *cx = col[group][0], *cy = col[group][1], *tc = col[group][2], *ts = col[group][3];
    const float inv = (float)(1.0 / binsize);
    const int tiles = (n_chains + kPairTile - 1) / kPairTile;
    const long long n_tiles = (long long)tiles * (tiles + 1) / 2 * slices;
    const int width = kPairTile / slices;
    for (long long t0 = (long long)blockIdx.x * kPairGroups; t0 < n_tiles; t0 += (long long)gridDim.x * kPairGroups) {
        const long long item = t0 + group, t = item / slices;
        const int k0 = (int)(item % slices) * width;  // the first of this slice's columns
        // tile t of the lower triangle -> (I, J), J <= I
        long long I = (long long)((sqrt(1.0 + 8.0 * (double)t) - 1.0) * 0.5);
        while (I * (I + 1) / 2 > t) I--;
        while ((I + 1) * (I + 2) / 2 <= t) I++;
        const long long J = t - I * (I + 1) / 2;
        const long long i = I * kPairTile + lane, j0 = J * kPairTile;
        __syncthreads();  // the previous columns are done with
        if (item < n_tiles && j0 + lane < n_chains) {
            const size_t j = (size_t)(j0 + lane) * 2;
            col[group][0][lane] = com[j];
            col[group][1][lane] = com[j + 1];
            if (kind != 0) {
                col[group][2][lane] = trig[j];
                col[group][3][lane] = trig[j + 1];
            }
        }
        __syncthreads();
        if (item >= n_tiles || i >= n_chains) continue;
        const double x = com[(size_t)i * 2], y = com[(size_t)i * 2 + 1];
        const double ca = kind != 0 ? trig[(size_t)i * 2] : 0.0, sa = kind != 0 ? trig[(size_t)i * 2 + 1] : 0.0;
        const int cols = (int)min((long long)kPairTile, i - j0);  // the columns below the diagonal
        const int k1 = min(cols, k0 + width);
        for (int k = k0; k < k1; k++) {
            const double s0 = centre_sep(x, cx[k], L), s1 = centre_sep(y, cy[k], L);
            const long long bin = pair_bin(__dadd_rn(__dmul_rn(s0, s0), __dmul_rn(s1, s1)), binsize, inv);
            if (bin < 0 || bin >= n_bins) continue;  // past the last bin of the reference's range
            atomicAdd(hc + bin, 2u);
            if (kind != 0) {
                double f = __dadd_rn(__dmul_rn(ca, tc[k]), __dmul_rn(sa, ts[k]));
                if (kind == 2) f = fabs(f);
                const long long fx = __double2ll_rn(2.0 * f * kFix);
                atomicAdd(hs + bin, (unsigned long long)fx);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_bins; i += blockDim.x) {
        if (hc[i]) atomicAdd(counts + i, (unsigned long long)hc[i]);
        if (kind != 0 && hs[i]) atomicAdd(sums + i, hs[i]);
    }
}

cudaError_t launch_chain_frames(int dim, int precision, const SysP &p, const int32_t *chain_start, double *com,
                                double *phi, int sym, double *trig, cudaStream_t st)
{
    const unsigned g = (unsigned)((p.n_chains + 63) / 64);
    if (dim == 2) {
        if (precision == 0)
            k_chain_frame<2, double><<<g, 64, 0, st>>>(p.pos, (const double *)p.tan, chain_start, p.n_chains, p.L, com,
                                                       phi, sym, trig);
        else
            k_chain_frame<2, float><<<g, 64, 0, st>>>(p.pos, (const float *)p.tan, chain_start, p.n_chains, p.L, com,
                                                      phi, sym, trig);
    } else {
        if (precision == 0)
            k_chain_frame<3, double><<<g, 64, 0, st>>>(p.pos, (const double *)p.tan, chain_start, p.n_chains, p.L, com,
                                                       phi, sym, trig);
        else
            k_chain_frame<3, float><<<g, 64, 0, st>>>(p.pos, (const float *)p.tan, chain_start, p.n_chains, p.L, com,
                                                      phi, sym, trig);
    }
    return cudaGetLastError();
}

cudaError_t launch_pair_corr(const double *com, const double *trig, int n_chains, double L, double binsize, int n_bins,
                             int kind, unsigned long long *counts, unsigned long long *sums, int sm_count,
                             cudaStream_t st)
{
    const size_t smem = (size_t)n_bins * ((kind != 0 ? sizeof(unsigned long long) : 0) + sizeof(unsigned));
    if (smem > 40 * 1024) {
        // the limit is every caller's: always that of the largest histogram
        const int limit = kMaxCorrBins * (int)(sizeof(unsigned long long) + sizeof(unsigned));
        cudaError_t e = cudaFuncSetAttribute(k_pair_corr, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
        if (e != cudaSuccess) return e;
    }
    const long long tiles = (n_chains + kPairTile - 1) / kPairTile;
    // no more slices than fill two CTAs on each SM: 1400 and 1500 chains 348 and
    // 458 us, 364 and 497 at one, the same at four
    int slices = 1;
    while (slices < kPairSlices && tiles * (tiles + 1) / 2 * slices <= (long long)kPairGroups * sm_count)
        slices *= 2;
    const long long n_tiles = tiles * (tiles + 1) / 2 * slices, groups = (n_tiles + kPairGroups - 1) / kPairGroups;
    // few CTAs, as each adds its histogram to the result; enough that a CTA's
    // 32-bit counts hold its pairs (2 * kPairTile^2 a whole tile: 2^18 of them)
    long long blocks = groups > 4LL * sm_count ? 4LL * sm_count : groups;
    blocks = blocks > n_tiles / 262144 + 1 ? blocks : n_tiles / 262144 + 1;
    k_pair_corr<<<(unsigned)blocks, kPairTile * kPairGroups, smem, st>>>(com, trig, n_chains, L, binsize, n_bins, kind,
                                                                         slices, counts, sums);
    return cudaGetLastError();
}

}  // namespace gcr
