// f8_sor.cuh — the red-black SOR pressure solve (poisson, fenep.f90:848-905) as
// one kernel: all sweeps, the residual sums and the stopping test on the device.
//
// A sweep of a small grid takes a microsecond or two; launched one by one, an
// iteration was four to seven kernels (two colours, boundary passes, two
// reduction stages) plus a host check every 25 iterations: 21 us an iteration on
// 64 x 32 x 32 in FP32, 45 in FP64.  Here the blocks meet at a barrier after each colour.  The
// neighbours are read through the wrap (periodic) or as the cell itself (the
// Neumann copy at a wall), which is what the boundary passes wrote between the
// sweeps, so the iterates are the same.
//
// Two forms:
//  * k_sor_cluster (FP32, up to SOR_CLUSTER_CELLS cells): a thread-block cluster
//    of up to 16 CTAs holds Phi in its shared memory in slabs of z planes with a
//    copy of the two neighbour planes, which their owners write through
//    distributed shared memory; the barrier is the cluster's hardware one.
//    64 x 32 x 32: 3.0 us an iteration, about 1 of it the barriers and the stopping
//    test (3.5 with the neighbours' rows read through distributed shared memory,
//    7.5 with all values in L2; 256 threads 3.4, 1024 threads 3.3).
//  * k_sor_grid: a cooperative grid of one CTA per SM over L2 (__ldcg) with a
//    counter in global memory.  Each wait is bounded (about a second): a wait
//    that runs out raises flag[2] and every block leaves.  64^3: 6.5 us an
//    iteration in FP32 (26 before), 16.7 in FP64 (82 before).  FP64 always takes
//    it (its sweeps are bound by the FP64 pipes of all SMs), and so do large
//    grids and those with too few planes to split.
#pragma once
#include <algorithm>
#include "f8_common.cuh"
#include "f8_df64.cuh"
#include "f8_recip.cuh"

namespace f8 {

constexpr long long SOR_WAIT_CYCLES = 2000000000LL;
constexpr int SOR_THREADS = 1024;
constexpr int SOR_CLUSTER_THREADS = 512;
constexpr int SOR_MAX_BLOCKS = 1024;    // partial sums per colour pair

// sums of squared residuals: FP64 residuals in FP64; FP32 residuals (24 bits
// each) as double-float, whose 48 bits are far below the residuals' own rounding
// and keep the FP64 pipe out of the sweep.  A square has twice the exponent, so
// FP32 residuals are scaled by a power of two first (sor_scale).
template <typename T>
struct SorSum;
template <>
struct SorSum<double> {
    double v;
    __device__ __forceinline__ void clear() { v = 0.0; }
    __device__ __forceinline__ void add_sq(double e) { v = v + e * e; }
    __device__ __forceinline__ void add(const SorSum &o) { v = v + o.v; }
    __device__ __forceinline__ SorSum shfl(int o) const { return SorSum{__shfl_xor_sync(0xffffffffu, v, o)}; }
    __device__ __forceinline__ double value() const { return v; }
};
template <>
struct SorSum<float> {
    df v;
    __device__ __forceinline__ void clear() { v = df{0.0f, 0.0f}; }
    __device__ __forceinline__ void add_sq(float e) {
        const float p = __fmul_rn(e, e);
        v = df_add(v, df{p, __fmaf_rn(e, e, -p)});
    }
    __device__ __forceinline__ void add(const SorSum &o) { v = df_add(v, o.v); }
    __device__ __forceinline__ SorSum shfl(int o) const {
        return SorSum{df{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)}};
    }
    __device__ __forceinline__ double value() const { return (double)v.hi + (double)v.lo; }
};
template <typename T>
__device__ __forceinline__ SorSum<T> warp_sum(SorSum<T> s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s.add(s.shfl(o));
    return s;
}

template <typename T>
struct SorArgs {
    T *Phi;                 // halo layout; interior read and written
    const T *R;             // interior right-hand side
    const double *er0;      // sum of R^2 (the reference's zero guard applied)
    SorSum<T> *part;        // SOR_MAX_BLOCKS partial sums, twice
    int *flag;              // [0] converged, [1] iteration, [2] a barrier wait ran out,
                            // [3] arrivals at the grid barrier; zero at launch
    T om, bx, by, bz, b0;   // relaxation, 1/dX^2 ..., the diagonal
    Recip rb0;              // 1/b0 (FP64)
    double eps;
    int itrmax, lgx, lgy;   // log2 of nx / 2 and ny
    long long wait = SOR_WAIT_CYCLES;   // limit of each wait of the grid barrier, clock cycles
};

// the residual, summed in the reference's order (fenep.f90:885-893); FP32: with
// the products fused into the sum, the same in both forms of the kernel
__device__ __forceinline__ double sor_residual(const SorArgs<double> &a, double zm, double ym, double xm, double p0,
                                               double xp, double yp, double zp, double f) {
    return a.bz * zm + a.by * ym + a.bx * xm - a.b0 * p0 + a.bx * xp + a.by * yp + a.bz * zp - f;
}
__device__ __forceinline__ float sor_residual(const SorArgs<float> &a, float zm, float ym, float xm, float p0, float xp,
                                              float yp, float zp, float f) {
    float e = __fmaf_rn(a.bz, zm, __fmul_rn(a.by, ym));
    e = __fmaf_rn(a.bx, xm, e);
    e = __fmaf_rn(-a.b0, p0, e);
    e = __fmaf_rn(a.bx, xp, e);
    e = __fmaf_rn(a.by, yp, e);
    return __fsub_rn(__fmaf_rn(a.bz, zp, e), f);
}
__device__ __forceinline__ float sor_update(float phi, float e, const SorArgs<float> &a) {
    return __fadd_rn(phi, __fmul_rn(a.om, e) / a.b0);
}
// the division by the known divisor b0 from its two-part reciprocal
__device__ __forceinline__ double sor_update(double phi, double e, const SorArgs<double> &a) {
    return phi + div_by(a.om * e, a.rb0);
}

// block sum in thread 0's warp (lane 0 of warp 0 holds it)
template <typename T>
__device__ __forceinline__ SorSum<T> block_sum(SorSum<T> s, SorSum<T> *sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s = warp_sum(s);
    if (lane == 0) sh[warp] = s;
    __syncthreads();
    if (warp == 0) {
        s.clear();
        if (lane < (int)(blockDim.x >> 5)) s = sh[lane];
        s = warp_sum(s);
    }
    return s;
}

// The power of two that takes sqrt(er0) into [1, 2): FP32 residuals down to
// 1e-19 of sqrt(er0) square without underflow, and one whose square overflows is
// 1e19 above it, far from converged (the sum is not below any bound then).  The
// scaling is exact, so the test is that of the plain squares wherever those are
// in range.
template <typename T>
__device__ __forceinline__ T sor_scale(double er0) {
    if constexpr (sizeof(T) == 8) {
        return 1.0;
    } else {
        const int e = ((__double2hiint(er0) >> 20) & 0x7ff) - 1023;
        return __int_as_float((127 - max(-126, min(126, e >> 1))) << 23);
    }
}

// sqrt(sum / er0) < eps: squared away from the boundary (eps >= 0)
__device__ __forceinline__ bool sor_done(double sum, double er0, double eps) {
    const double e2 = eps * eps * er0;
    if (sum < e2 * (1.0 - 1.0e-12)) return true;
    return !(sum > e2 * (1.0 + 1.0e-12)) && sqrt(sum / er0) < eps;
}

// true when the wait ran out
__device__ __forceinline__ bool sor_grid_barrier(unsigned *bar, unsigned &arrivals, int *late, long long wait) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        arrivals += gridDim.x;
        __threadfence();
        atomicAdd(bar, 1u);
        const long long t0 = clock64();
        unsigned v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (behind(v, arrivals) && clock64() - t0 > wait) { *late = 1; break; }
        } while (behind(v, arrivals));
    }
    __syncthreads();
    return *late != 0;
}

template <typename T>
__global__ void __launch_bounds__(SOR_THREADS, 1) k_sor_grid(SorArgs<T> a, Geo g) {
    __shared__ SorSum<T> sh[32];
    __shared__ int late, stop;
    if (threadIdx.x == 0) late = stop = 0;
    __syncthreads();
    const int n = (g.nx >> 1) * g.ny * g.nz, stride = gridDim.x * blockDim.x;
    const int oy = g.sx, oz = g.sx * g.sy;
    const T sc = sor_scale<T>(*a.er0);
    const double er0 = *a.er0 * ((double)sc * (double)sc);
    unsigned arrivals = 0, *bar = reinterpret_cast<unsigned *>(a.flag + 3);
    for (int itr = 1; itr <= a.itrmax; ++itr) {
        SorSum<T> s;
        s.clear();
#pragma unroll 1
        for (int color = 0; color < 2; ++color) {
            for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += stride) {
                const int row = c >> a.lgx, j = (row & (g.ny - 1)) + 1, k = (row >> a.lgy) + 1;
                const int i = 2 * (c & ((1 << a.lgx) - 1)) + 1 + ((j + k + 1 + color) & 1);
                const int h = hix(g, i, j, k), q = qix(g, i, j, k);
                const T *P = a.Phi + h;
                // wrapped neighbours; at a wall the cell itself, in 2D no z neighbour
                const int xm = i > 1 ? -1 : g.nx - 1, xp = i < g.nx ? 1 : 1 - g.nx;
                const int ym = j > 1 ? -oy : (g.walls ? 0 : (g.ny - 1) * oy), yp = j < g.ny ? oy : (g.walls ? 0 : (1 - g.ny) * oy);
                const int zm = k > 1 ? -oz : (g.nz - 1) * oz, zp = k < g.nz ? oz : (1 - g.nz) * oz;
                const T p0 = __ldcg(P);
                const T e = sor_residual(a, __ldcg(P + zm), __ldcg(P + ym), __ldcg(P + xm), p0, __ldcg(P + xp),
                                         __ldcg(P + yp), __ldcg(P + zp), a.R[q]);
                s.add_sq(e * sc);
                __stcg(a.Phi + h, sor_update(p0, e, a));
            }
            if (color == 0 && sor_grid_barrier(bar, arrivals, &late, a.wait)) break;
        }
        // the block's sum, then every block's in the same order
        s = block_sum(s, sh);
        SorSum<T> *part = a.part + (itr & 1) * SOR_MAX_BLOCKS;
        if (threadIdx.x == 0) part[blockIdx.x] = s;
        if (late || sor_grid_barrier(bar, arrivals, &late, a.wait)) {
            if (threadIdx.x == 0) a.flag[2] = 1;
            return;
        }
        if (threadIdx.x < 32) {
            SorSum<T> t;
            t.clear();
            for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) {
                SorSum<T> p;
                if constexpr (sizeof(T) == 8) {
                    p.v = __ldcg(&part[b].v);
                } else {
                    const float2 f = __ldcg(reinterpret_cast<const float2 *>(&part[b]));
                    p.v = df{f.x, f.y};
                }
                t.add(p);
            }
            t = warp_sum(t);
            if (threadIdx.x == 0) {
                const bool done = sor_done(t.value(), er0, a.eps);
                stop = done;
                if (blockIdx.x == 0 && (done || itr == a.itrmax)) {
                    a.flag[1] = itr;
                    a.flag[0] = done;
                }
            }
        }
        __syncthreads();
        if (stop) return;
    }
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, float a, float b) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned addr, float a) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(a) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// SLOTS: cell pairs (x neighbours, one of each colour) per thread, whose values
// and right-hand sides stay in registers.  A CTA owns nz / gridDim.x planes;
// shared memory holds them between copies of the plane below and above (rows of
// the even cells, then the odd ones, so that a warp's accesses are consecutive).
template <int SLOTS>
__global__ void __launch_bounds__(SOR_CLUSTER_THREADS, 1) k_sor_cluster(SorArgs<float> a, Geo g) {
    extern __shared__ float phi[];
    __shared__ SorSum<float> sh[32];
    __shared__ float2 part[3][16];
    __shared__ float shf[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nx = g.nx, half = nx >> 1, ncta = gridDim.x;
    const int planes = g.nz / ncta, plane = nx * g.ny, pairs = planes * plane >> 1;
    const unsigned rank = cluster_rank(), base = (unsigned)__cvta_generic_to_shared(phi);
    const unsigned pbase = (unsigned)__cvta_generic_to_shared(&part[0][0]);
    const unsigned prev = rank == 0 ? ncta - 1 : rank - 1, next = rank == ncta - 1u ? 0 : rank + 1;
    for (int q = threadIdx.x; q < (planes + 2) * plane; q += blockDim.x) {
        const int i = q % nx, row = q / nx, j = row % g.ny;
        int k = (int)rank * planes + row / g.ny - 1;
        k = k < 0 ? k + g.nz : (k >= g.nz ? k - g.nz : k);
        phi[row * nx + (i & 1) * half + (i >> 1)] = __ldcg(a.Phi + hix(g, i + 1, j + 1, k + 1));
    }
    __syncthreads();
    int row_[SLOTS], up[SLOTS], dn[SLOTS];      // the pair's row, its y neighbours' offsets
    int par[SLOTS];                             // parity, or -1 for no pair
    unsigned push[SLOTS][2];                    // where the copies of its row lie in the previous / next CTA (0: none)
    float pv[SLOTS][2], rv[SLOTS][2];
    const int ix = threadIdx.x & (half - 1);    // SOR_CLUSTER_THREADS is a multiple of half (a power of two up to 512)
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        const int c = threadIdx.x + s * SOR_CLUSTER_THREADS, rl = c >> a.lgx;
        const int j = rl & (g.ny - 1), kl = rl >> a.lgy, k = (int)rank * planes + kl;
        par[s] = c < pairs ? (j + k + 1) & 1 : -1;
        row_[s] = (c < pairs ? rl + g.ny : g.ny) * nx;
        up[s] = j < g.ny - 1 ? nx : (g.walls ? 0 : (1 - g.ny) * nx);
        dn[s] = j > 0 ? -nx : (g.walls ? 0 : (g.ny - 1) * nx);
        push[s][0] = c < pairs && kl == 0 ? mapa(base + 4u * (unsigned)((planes + 1) * plane + j * nx), prev) : 0u;
        push[s][1] = c < pairs && kl == planes - 1 ? mapa(base + 4u * (unsigned)(j * nx), next) : 0u;
#pragma unroll
        for (int color = 0; color < 2; ++color) {
            const int o = par[s] ^ color;
            pv[s][color] = rv[s][color] = 0.0f;
            if (par[s] >= 0) {
                pv[s][color] = phi[row_[s] + o * half + ix];
                rv[s][color] = a.R[((size_t)k * g.ny + j) * nx + 2 * ix + o];
            }
        }
    }
    cluster_barrier();
    const float sc = sor_scale<float>(*a.er0);
    const double er0 = *a.er0 * ((double)sc * (double)sc);
    const float above = (float)(a.eps * a.eps * er0) * 1.0001f;
    for (int itr = 1; itr <= a.itrmax; ++itr) {
        SorSum<float> s;
        s.clear();
#pragma unroll
        for (int color = 0; color < 2; ++color) {
#pragma unroll
            for (int t = 0; t < SLOTS; ++t) {
                if (par[t] < 0) continue;
                const int o = par[t] ^ color;
                const float *own = phi + row_[t], *at = own + o * half + ix;
                // x neighbours: the pair's other cell and the next pair's
                const float xi = own[(o ? 0 : half) + ix], xo = own[o ? ((ix + 1) & (half - 1)) : half + ((ix - 1) & (half - 1))];
                const float xm = o ? xi : xo, xp = o ? xo : xi;
                const float p0 = pv[t][color];
                const float ym = dn[t] ? at[dn[t]] : p0, yp = up[t] ? at[up[t]] : p0;
                const float e = sor_residual(a, at[-plane], ym, xm, p0, xp, yp, at[plane], rv[t][color]);
                s.add_sq(e * sc);
                const float v = sor_update(p0, e, a);
                pv[t][color] = v;
                phi[row_[t] + o * half + ix] = v;
                const unsigned ofs = 4u * (unsigned)(o * half + ix);
                if (push[t][0]) st_cluster(push[t][0] + ofs, v);
                if (push[t][1]) st_cluster(push[t][1] + ofs, v);
            }
            if (color == 0) cluster_barrier();
        }
        // The stopping test first on FP32 sums (relative error below 1e-4): far
        // above the boundary, as nearly always, the double-float sum is not needed.
        // Every warp reduces the CTAs' values itself.
        float f = s.v.hi;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
        if (lane == 0) shf[warp] = f;
        __syncthreads();
        if (warp == 0) {
            f = lane < SOR_CLUSTER_THREADS / 32 ? shf[lane] : 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
            if (lane < ncta) st_cluster(mapa(pbase + 8u * (16u * (itr & 1) + rank), lane), f, 0.0f);
        }
        cluster_barrier();
        f = lane < ncta ? part[itr & 1][lane].x : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
        if (f > above && itr < a.itrmax) continue;
        // the double-float sum (uniform over the cluster: f is the same everywhere)
        s = block_sum(s, sh);
        if (warp == 0 && lane < ncta) st_cluster(mapa(pbase + 8u * (32u + rank), lane), s.v.hi, s.v.lo);
        cluster_barrier();
        s.clear();
        if (lane < ncta) s.v = df{part[2][lane].x, part[2][lane].y};
        s = warp_sum(s);
        const bool done = sor_done(s.value(), er0, a.eps);
        if (rank == 0 && threadIdx.x == 0 && (done || itr == a.itrmax)) {
            a.flag[1] = itr;
            a.flag[0] = done;
        }
        if (done) break;
        cluster_barrier();   // part[2] and sh are free again
    }
    // no remote access follows the last cluster barrier
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        const int c = threadIdx.x + s * SOR_CLUSTER_THREADS, rl = c >> a.lgx;
        if (par[s] < 0) continue;
        float *out = a.Phi + hix(g, 2 * ix + 1, (rl & (g.ny - 1)) + 1, (int)rank * planes + (rl >> a.lgy) + 1);
        out[par[s]] = pv[s][0];
        out[par[s] ^ 1] = pv[s][1];
    }
}

// Grids of up to this many cells (8 cell pairs a thread of 16 CTAs) take the
// cluster, larger ones all SMs: 64^3 6.5 us an iteration there.  Against sweeps
// launched one by one (150 of them, FP32): 64^3 4.0 -> 1.15 ms, 128^3 7.9 -> 2.95,
// 256x128x128 11.8 -> 5.0.
constexpr long SOR_CLUSTER_CELLS = 131072;
constexpr int SOR_CLUSTER_SMEM = 200 * 1024;

// the largest cluster of these blocks that the device can hold (8 is portable;
// 16 where a GPC has the SMs)
inline cudaError_t sor_cluster_size(int *out) {
    *out = 8;
    for (auto *k : {k_sor_cluster<1>, k_sor_cluster<2>, k_sor_cluster<4>, k_sor_cluster<8>}) {
        F8_CUDA_RET(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        F8_CUDA_RET(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SOR_CLUSTER_SMEM));
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(SOR_CLUSTER_THREADS);
    cfg.dynamicSmemBytes = SOR_CLUSTER_SMEM;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_sor_cluster<8>, &cfg) == cudaSuccess && n > 0) *out = 16;
    else cudaGetLastError();
    return cudaSuccess;
}

// the sweeps of one solve on stream s (the flags are cleared here);
// max_cluster > 1 allows the cluster form
template <typename T>
inline cudaError_t sor_sweeps(SorArgs<T> a, const Geo &g, int sms, int max_cluster, cudaStream_t s) {
    // no sum passes a test against a negative or NaN tolerance, nor against zero:
    // all itrmax sweeps run
    if (!(a.eps > 0.0)) a.eps = 0.0;
    a.lgx = a.lgy = 0;
    while ((2 << a.lgx) < g.nx) ++a.lgx;
    while ((1 << a.lgy) < g.ny) ++a.lgy;
    F8_CUDA_RET(cudaMemsetAsync(a.flag, 0, 4 * sizeof(int), s));
    const long n = (long)g.nx * g.ny * g.nz, need = (n / 2 + SOR_CLUSTER_THREADS - 1) / SOR_CLUSTER_THREADS;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cfg.blockDim = dim3(SOR_THREADS);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if constexpr (sizeof(T) == 4) {
        int cl = 1;
        while (cl < max_cluster && cl < need && cl < g.nz) cl *= 2;
        const int slots = (int)((n / 2 / cl + SOR_CLUSTER_THREADS - 1) / SOR_CLUSTER_THREADS);
        const size_t smem = (size_t)(g.nz / cl + 2) * g.nx * g.ny * sizeof(float);
        if (max_cluster > 1 && n <= SOR_CLUSTER_CELLS && slots <= 8 && smem <= SOR_CLUSTER_SMEM) {
            cfg.gridDim = dim3(cl);
            cfg.blockDim = dim3(SOR_CLUSTER_THREADS);
            cfg.dynamicSmemBytes = smem;
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = cl;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            count_launch();
            if (slots <= 1) return cudaLaunchKernelEx(&cfg, k_sor_cluster<1>, a, g);
            if (slots <= 2) return cudaLaunchKernelEx(&cfg, k_sor_cluster<2>, a, g);
            if (slots <= 4) return cudaLaunchKernelEx(&cfg, k_sor_cluster<4>, a, g);
            return cudaLaunchKernelEx(&cfg, k_sor_cluster<8>, a, g);
        }
    }
    // every SM its share, in as many threads as it has cells of a colour
    const int blocks = (int)std::min<long>((n / 2 + 31) / 32, std::min(sms, SOR_MAX_BLOCKS));
    const long share = (n / 2 + blocks - 1) / blocks;
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)std::min<long>((share + 31) / 32 * 32, SOR_THREADS));
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, k_sor_grid<T>, a, g);
}

}  // namespace f8
