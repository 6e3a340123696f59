// f8_codes_fp64.cu — the SPD face-candidate choice of the FP64 3D step
// (CpxCnx .. CpzCnz, fenep.f90:169-242 with the Vieta test 425-444), decided
// on the FP32 pipes wherever rounding cannot change it.
//
// The choice compares the least eigenvalues of six candidate faces per
// direction, 18 evaluations of Vieta's formula per cell.  In FP64 each costs
// about 170 pipe slots, and one FP64 warp instruction occupies its SM
// sub-partition for 64 cycles (measured: 0.55e12 operations/s on the chip).
// Only the comparison leaves the kernel, so k_codes3_filter evaluates the
// faces in double-float arithmetic (f8_df64.cuh) with an error bound that
// covers its own rounding and that of the FP64 formula.  Where the best
// candidate leads by more than the bounds, the FP64 evaluation makes the same
// choice; every other (cell, direction) is queued and k_codes3_exact
// (f8_step_fp64.cu) evaluates the FP64 formula itself.  The codes are therefore
// those of the FP64 evaluation, bit for bit.
//
// Bounds, for a face with mean m, p = |B|^2 / 6 of its deviator B, s = sqrt(p),
// r = det(B) / (2 s^3), u = sqrt(1 - r) and lambda = m + s 2t(u) (the smallest
// root of 4t^3 - 3t = r, |t| <= 1):
//  * the products of p and det(B) in double-float carry an absolute error of some
//    1e-12 of their scale, given B, which moves lambda by at most 1e-11 s / u;
//  * B itself: C's components are split to 48 bits before the mean is taken off, and
//    the differences and means round to as many.  The components of the cell and its
//    neighbours reach a few M (M = |m| + 2s), so that is up to 10 x 2^-48 M in each
//    component of B (160 eps M, eps = 2^-52).  It changes s by as much and r by
//    6 x 160 eps M / s, so lambda by 160 eps M (4 + 2.5 / u);
//  * the FP32 evaluation of u, 2t(u) (polynomial error 2.2e-7) and the sum moves
//    it by at most 4e-6 s + 1e-6 |m - m0| (m0 the cell's mean, common to every
//    face and left out of the comparisons);
//  * the FP64 formula forms p = a1 - a2^2/3 and q from the unshifted
//    components, with errors up to ~20 eps M^2 and ~100 eps M^3; they move lambda
//    by at most eps M (M/s) (20 + 26 (M/s)/u);
//  * M/s is at least 2, so this and the error of B together stay below
//    eps M (M/s) (340 + 126 (M/s)/u): 1e-13 M (M/s) (1 + (M/s)/u), 450 eps, is above;
//  * the sentinel for repeated roots (|r| >= 1 as FP64 rounds it) can differ
//    only where 1 - r^2 is within 4e-8 + 4e-13 (M/s)^3 of zero (1800 eps (M/s)^3: the
//    FP64 formula's 2 |dr| is 100 eps (M/s)^3 + 60 eps (M/s)^2, B's 1920 eps M/s):
//    such faces, and any that over- or underflow to NaN, are queued.
#include <cuda_runtime.h>
#include "f8_codes_filter.cuh"
#include "f8_common.cuh"
#include "f8_kernels.h"

namespace f8 {
namespace {

constexpr int FILTER_THREADS = 256;

// C (FP64) -> double-float pairs, four values a thread; clears the queue
__global__ void __launch_bounds__(256) k_split_c(const double2 *__restrict__ C, float4 *__restrict__ out, int n2,
                                                 int *__restrict__ count) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < 3) count[q] = 0;
    if (q >= n2) return;
    const double2 v = C[q];
    const df a = df_from_d(v.x), b = df_from_d(v.y);
    out[q] = make_float4(a.hi, a.lo, b.hi, b.lo);
}

// The candidate code of every direction of a cell (0..3), or the cell's place
// in the queue of that direction.  Bound by the packed FP32 pipe (about 4,000
// instructions a cell, 136 registers).  Split, filter and exact kernel together,
// a developed flow: 64^3 143 us (all cells in FP64: 1992), a 128x64x64 channel
// 301 us (3805).  Near C = I, where FP64's own cancellation decides, nearly every
// cell is queued and the stage takes what the FP64 evaluation takes.
__global__ void __launch_bounds__(FILTER_THREADS) k_codes3_filter(const float2 *__restrict__ C,
                                                                  uint8_t *__restrict__ codes,
                                                                  uint8_t *__restrict__ codes_g, Geo g, int cs,
                                                                  unsigned *__restrict__ q0, unsigned *__restrict__ q1,
                                                                  unsigned *__restrict__ q2, int *__restrict__ count) {
    __shared__ int need[3], base[3];
    const int tid = threadIdx.x + 32 * threadIdx.y;
    if (tid < 3) need[tid] = 0;
    __syncthreads();
    const int i = blockIdx.x * 32 + threadIdx.x + 1;
    const int j = blockIdx.y * (FILTER_THREADS / 32) + threadIdx.y + prow0(g);
    const int k = blockIdx.z + 1;
    const bool active = i <= g.nx && j < prow0(g) + prows(g);
    int code = 0, slot[3] = {-1, -1, -1};
    if (active) {
        const int h = hix(g, i, j, k);
        codes::CellC c;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const float2 v = C[(size_t)m * cs + h];
            c.c[m] = df{v.x, v.y};
        }
        codes::cell_split(c);
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            const int od = d == 0 ? 1 : (d == 1 ? g.sx : g.sx * g.sy);
            // beyond the ghost rows of a wall channel C is zero
            const bool lo = !(d == 1 && j == 0), hi = !(d == 1 && j == g.ny + 1);
            df2 dv[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const float2 *Cm = C + (size_t)m * cs + h;
                const float2 cm = lo ? Cm[-od] : make_float2(0.0f, 0.0f), cp = hi ? Cm[od] : make_float2(0.0f, 0.0f);
                dv[m] = df2_sub(df2{make_float2(c.c[m].hi, cp.x), make_float2(c.c[m].lo, cp.y)},
                                df2{make_float2(cm.x, c.c[m].hi), make_float2(cm.y, c.c[m].lo)});
            }
            const int r = codes::choose(c, dv);
            if (r >= 0) {
                code |= r << (2 * d);
            } else {
                const int at = atomicAdd(&need[d], 1);
                if (d == 0) slot[0] = at;
                else if (d == 1) slot[1] = at;
                else slot[2] = at;
            }
        }
        uint8_t *dst = (j >= 1 && j <= g.ny) ? codes + qix(g, i, j, k) : codes_g + gcix(g, i, j, k);
        *dst = (uint8_t)code;
    }
    __syncthreads();
    if (tid < 3 && need[tid]) base[tid] = atomicAdd(&count[tid], need[tid]);
    __syncthreads();
    if (active) {
        const unsigned e = (unsigned)(i - 1) + (unsigned)g.nx * ((unsigned)(j - prow0(g)) + (unsigned)prows(g) * (unsigned)(k - 1));
        if (slot[0] >= 0) q0[base[0] + slot[0]] = e;
        if (slot[1] >= 0) q1[base[1] + slot[1]] = e;
        if (slot[2] >= 0) q2[base[2] + slot[2]] = e;
    }
}

}  // namespace

// C as double-float pairs goes to the C buffer of the next update (not yet
// written there), the queues hold one entry per cell and direction at most.
cudaError_t codes3_filter(Dev &d, cudaStream_t s) {
    const Geo &g = d.g;
    const int n2 = d.cs / 2 * 6;   // cs is even (sx is)
    float2 *cdf = reinterpret_cast<float2 *>(d.Cn);
    k_split_c<<<(n2 + 255) / 256, 256, 0, s>>>(reinterpret_cast<const double2 *>(d.C), reinterpret_cast<float4 *>(cdf),
                                               n2, d.code_count); count_launch();
    const dim3 blk(32, FILTER_THREADS / 32);
    const dim3 grd((g.nx + 31) / 32, (prows(g) + blk.y - 1) / blk.y, g.nz);
    k_codes3_filter<<<grd, blk, 0, s>>>(cdf, d.codes, d.codes_g, g, d.cs, codes3_queue(d, 0), codes3_queue(d, 1),
                                        codes3_queue(d, 2), d.code_count); count_launch();
    return cudaGetLastError();
}

}  // namespace f8
