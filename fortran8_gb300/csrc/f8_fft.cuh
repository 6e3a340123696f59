// f8_fft.cuh — batched radix-2 Stockham FFT kernels and the wall-normal
// tridiagonal solve, templated on the real type.
//
// Replaces FFTW (fft_solve, fenep.f90:1400-1428; fenep_2d.f90:841-867) and the
// Thomas solver tdma (fenep_2d.f90:1145-1177).  Every butterfly is written in
// the same order as the CPU oracle's Stockham loop, so the FP64 instantiation
// compiled without FMA contraction reproduces the oracle bit for bit.
//
// Spectral layout: complex values interleaved (re, im), [k][j][kx] with
// kx = 0..NX/2 (NXH = NX/2+1 values per row).
#pragma once
#include <algorithm>
#include <type_traits>
#include "f8_common.cuh"
#include "f8_df64.cuh"
#include "f8_recip.cuh"

namespace f8 {

template <typename T>
struct Cx { T r, i; };

__host__ __device__ inline int ilog2_pow2(int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

// b * (wr, wi).  FP64: rounded products and sum, as the oracle forms them.  FP32:
// one product fused into the sum, in a fixed order so that every form of a
// transform gives the same bits; INV: the order of a conjugated twiddle.
template <bool INV>
__device__ __forceinline__ Cx<double> twiddle_mul(Cx<double> b, double wr, double wi) {
    return Cx<double>{__dsub_rn(__dmul_rn(b.r, wr), __dmul_rn(b.i, wi)), __dadd_rn(__dmul_rn(b.r, wi), __dmul_rn(b.i, wr))};
}
template <bool INV>
__device__ __forceinline__ Cx<float> twiddle_mul(Cx<float> b, float wr, float wi) {
    return Cx<float>{__fmaf_rn(b.r, wr, -__fmul_rn(b.i, wi)),
                     INV ? __fmaf_rn(b.i, wr, __fmul_rn(b.r, wi)) : __fmaf_rn(b.r, wi, __fmul_rn(b.i, wr))};
}

// One butterfly (index j of 2^(lg-1)) of the Stockham stage of span 2^ls on a
// line of 2^lg complex values in shared memory, x -> y.
//   tw: forward twiddles exp(-2 pi i t/n), t < n/2 (re, im arrays)
// The first stage's twiddle is 1.
template <bool INV, typename T>
__device__ __forceinline__ void stockham_stage(const Cx<T> *x, Cx<T> *y, int lg, int ls, int j, const T *twr,
                                               const T *twi, int sign) {
    const int half = 1 << (lg - 1), ns = 1 << ls;
    const int kk = j & (ns - 1);
    const Cx<T> a = x[j], b = x[j + half];
    Cx<T> t = b;
    if (ls > 0) {
        const int q = kk << (lg - 1 - ls);
        t = twiddle_mul<INV>(b, twr[q], sign < 0 ? twi[q] : -twi[q]);
    }
    const int o = ((j >> ls) << (ls + 1)) + kk;
    y[o].r = a.r + t.r; y[o].i = a.i + t.i;
    y[o + ns].r = a.r - t.r; y[o + ns].i = a.i - t.i;
}

// Shapes of the transform launches.  A block takes up to 256 butterflies of a
// stage (one per thread).  A small problem is bound by the chain of its stages
// (an FP64 butterfly holds a sub-partition's pipe for 640 cycles), not by
// memory, so its lines are spread over the chip: fewer lines per block until
// there are two blocks per SM (304).  2D 128^2, FP64: 19 us a pass with 16
// columns in each of 5 blocks, 4 us with one in each of 65.
constexpr long FFT_MIN_BLOCKS = 304;
constexpr long FFT_REG_WARPS = 150;

// lines (row pairs) per block of an x pass over `pairs` row pairs
inline int fft_pairs_per_block(int n, long pairs) {
    int p = std::max(1, 512 / n);
    while (p > 1 && p * n > 64 && (pairs + p - 1) / p < FFT_MIN_BLOCKS) p >>= 1;
    return p;
}

// columns per block of a line pass; segments of at least 32 bytes where the
// problem is large enough for memory to matter
template <typename T>
inline int fft_cols_per_block(int n, int ncols, long sets) {
    int tx = std::max(512 / n, (int)(32 / sizeof(Cx<T>)));
    while (tx > 1 && tx * n > 64 && (ncols + tx - 1) / tx * sets < FFT_MIN_BLOCKS) tx >>= 1;
    return tx;
}
template <typename T>
inline int fft_line_threads(int n, int tx) {
    return std::min(256, std::max(32, n / 2 * tx));
}

// ---------------------------------------------------------------------------
// A line of n = 2^LG values (32 .. 1024) held by G = n / 8 threads: the stages of
// the Stockham kernels below (the same butterflies, twiddles and order, so the
// same bits) as decimation in time, up to three of them at a time on eight
// values in registers, with one exchange through shared memory between the
// passes instead of one per stage.  The value of element e lies at ix(e); lanes
// of one line and neighbouring lines fall into distinct banks.
template <int LG>
struct LineFft {
    static constexpr int N = 1 << LG, G = N / 8, PITCH = N + N / 8 + 1;
    static __device__ __forceinline__ int ix(int e) { return e + (e >> 3); }
    static __device__ __forceinline__ int brev(int e) { return (int)(__brev((unsigned)e) >> (32 - LG)); }
};

// stages L0 .. L0 + R - 1 on the groups base + (s << L0), s < 2^R, of thread t
template <bool INV, int LG, int L0, int R, typename T, typename Load, typename Store>
__device__ __forceinline__ void fft_pass(int t, const T *twr, const T *twi, Load load, Store store) {
    constexpr int W = 1 << R, U = 8 / W;
    Cx<T> v[8];
    int lo[U], base[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int g = t + u * LineFft<LG>::G;
        lo[u] = g & ((1 << L0) - 1);
        base[u] = ((g >> L0) << (L0 + R)) | lo[u];
#pragma unroll
        for (int s = 0; s < W; ++s) v[u * W + s] = load(base[u] + (s << L0));
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const int m = 1 << a;
#pragma unroll
            for (int s = 0; s < W; ++s) {
                if (s & m) continue;
                const Cx<T> x = v[u * W + s], b = v[u * W + s + m];
                Cx<T> c = b;
                if (L0 > 0 || (s & (m - 1))) {       // the others' twiddle is 1
                    const int q = (lo[u] + ((s & (m - 1)) << L0)) << (LG - 1 - L0 - a);
                    c = twiddle_mul<INV>(b, twr[q], INV ? -twi[q] : twi[q]);
                }
                v[u * W + s] = Cx<T>{x.r + c.r, x.i + c.i};
                v[u * W + s + m] = Cx<T>{x.r - c.r, x.i - c.i};
            }
        }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int s = 0; s < W; ++s) store(base[u] + (s << L0), v[u * W + s]);
}

// natural order in (load(e)) and out (store(e, value)); z: the line's PITCH
// values of shared memory, free on entry.  Every thread of the block takes part.
template <bool INV, int LG, typename T, typename Load, typename Store>
__device__ __forceinline__ void fft_line(Cx<T> *z, int t, const T *twr, const T *twi, Load load, Store store) {
    using L = LineFft<LG>;
    auto get = [&](int e) { return z[L::ix(e)]; };
    auto put = [&](int e, Cx<T> v) { z[L::ix(e)] = v; };
    fft_pass<INV, LG, 0, 3, T>(t, twr, twi, [&](int e) { return load(L::brev(e)); }, put);
    __syncthreads();
    if constexpr (LG == 5) fft_pass<INV, LG, 3, 2, T>(t, twr, twi, get, store);
    else if constexpr (LG == 6) fft_pass<INV, LG, 3, 3, T>(t, twr, twi, get, store);
    else {
        constexpr int R1 = LG == 7 ? 2 : 3, L2 = 3 + R1;
        fft_pass<INV, LG, 3, R1, T>(t, twr, twi, get, put);
        __syncthreads();
        if constexpr (LG == 10) {
            fft_pass<INV, LG, 6, 2, T>(t, twr, twi, get, put);
            __syncthreads();
            fft_pass<INV, LG, 8, 2, T>(t, twr, twi, get, store);
        } else fft_pass<INV, LG, L2, LG - L2, T>(t, twr, twi, get, store);
    }
}

// Lines of 32 to 1024 values go through registers in FP32, and in FP64 where
// they make 150 warps or more: a smaller FP64 problem is a chain of stages,
// shortest with one butterfly per thread (f8_fft_solve, us, stages in shared
// memory / in registers: 128^2 46.5 / 68.8, 256^2 (128 warps) 55 / 78, 512^2 104 / 99,
// 64^3 119 / 115, 128x64x64 298 / 266, 256x128x128 1179 / 1100; batches of three
// 64^3 solves 79 / 76 each).  FP32 lines of 512: x pass 6.3 / 4.3, y lines with
// the division 11.4 / 9.8.
template <typename T>
inline bool fft_in_registers(int n, long lines) {
    if (n < 32 || n > 1024) return false;
    return sizeof(T) == 4 || lines * (n / 8) >= 32 * FFT_REG_WARPS;
}

// go(integral_constant LG) for a line of n = 2^LG values, 32 .. 1024
template <typename F>
inline void fft_by_length(int n, F go) {
    switch (n) {
    case 32: go(std::integral_constant<int, 5>{}); break;
    case 64: go(std::integral_constant<int, 6>{}); break;
    case 128: go(std::integral_constant<int, 7>{}); break;
    case 256: go(std::integral_constant<int, 8>{}); break;
    case 512: go(std::integral_constant<int, 9>{}); break;
    default: go(std::integral_constant<int, 10>{}); break;
    }
}

// Up to three transforms of the same shape in one launch (blockIdx.z; their
// spectra lie hstride values apart).
template <typename P>
struct Batch {
    P p[3];
};

// ---------------------------------------------------------------------------
// x direction, real <-> half spectrum, two rows per complex transform.
//
// Forward: rows (j0 + jj, j0 + jj + 1) of plane k of the interior-ordered
// source src (row length n, nrow_src rows per plane) become spectral rows
// jj, jj+1 of H (nrow_h rows per plane).  One CTA handles blockDim.x / (n/2) row
// pairs with n/2 threads each.
template <typename T, typename TS>
__global__ void k_fft_x_fwd(Batch<const TS *> srcs, T *__restrict__ H, size_t hstride, int lg, int nrow_src, int j0,
                            int nrow_h, int npairs_per_plane, int nplanes, const T *__restrict__ twr,
                            const T *__restrict__ twi) {
    extern __shared__ unsigned char smem_raw[];
    Cx<T> *sm = reinterpret_cast<Cx<T> *>(smem_raw);
    const int n = 1 << lg, half = n >> 1, tpp = half;
    const TS *__restrict__ src = srcs.p[blockIdx.z];
    H += (size_t)blockIdx.z * hstride;
    const int p = threadIdx.x >> (lg - 1), t = threadIdx.x & (half - 1);
    const long pair = (long)blockIdx.x * (blockDim.x >> (lg - 1)) + p;
    const bool active = pair < (long)npairs_per_plane * nplanes;
    Cx<T> *x = sm + (size_t)p * 2 * n, *y = x + n;
    int k = 0, jj = 0;
    if (active) {
        k = (int)(pair / npairs_per_plane);
        jj = 2 * (int)(pair % npairs_per_plane);
        const TS *ra = src + (size_t)n * ((size_t)(j0 + jj - 1) + (size_t)nrow_src * k);
        const TS *rb = ra + n;
        for (int e = t; e < n; e += tpp) { x[e].r = T(ra[e]); x[e].i = T(rb[e]); }
    }
    __syncthreads();
    for (int ls = 0; ls < lg; ++ls) {
        if (active) stockham_stage<false>(x, y, lg, ls, t, twr, twi, -1);
        __syncthreads();
        Cx<T> *tmp = x; x = y; y = tmp;
    }
    if (!active) return;
    const int nxh = half + 1;
    T *ha = H + 2 * ((size_t)nxh * ((size_t)jj + (size_t)nrow_h * k));
    T *hb = ha + 2 * nxh;
    for (int kx = t; kx < nxh; kx += tpp) {
        const Cx<T> zk = x[kx], zm = x[(n - kx) & (n - 1)];
        ha[2 * kx] = (zk.r + zm.r) * T(0.5);
        ha[2 * kx + 1] = (zk.i - zm.i) * T(0.5);
        hb[2 * kx] = (zk.i + zm.i) * T(0.5);
        hb[2 * kx + 1] = (zm.r - zk.r) * T(0.5);
    }
}

template <int LG, typename T, typename TS>
__global__ void __launch_bounds__(256) k_fft_x_fwd_r(Batch<const TS *> srcs, T *__restrict__ H, size_t hstride,
                                                     int nrow_src, int j0, int nrow_h, int npairs_per_plane, int nplanes,
                                                     const T *__restrict__ twr, const T *__restrict__ twi) {
    using L = LineFft<LG>;
    extern __shared__ unsigned char smem_raw[];
    const TS *__restrict__ src = srcs.p[blockIdx.z];
    H += (size_t)blockIdx.z * hstride;
    const int p = threadIdx.x / L::G, t = threadIdx.x % L::G;
    const long pair = (long)blockIdx.x * (blockDim.x / L::G) + p;
    const bool active = pair < (long)npairs_per_plane * nplanes;
    Cx<T> *z = reinterpret_cast<Cx<T> *>(smem_raw) + p * L::PITCH;
    const int k = active ? (int)(pair / npairs_per_plane) : 0, jj = active ? 2 * (int)(pair % npairs_per_plane) : 0;
    const TS *ra = src + (size_t)L::N * ((size_t)(j0 + jj - 1) + (size_t)nrow_src * k), *rb = ra + L::N;
    fft_line<false, LG, T>(z, t, twr, twi, [&](int e) { return active ? Cx<T>{T(ra[e]), T(rb[e])} : Cx<T>{T(0), T(0)}; },
                           [&](int e, Cx<T> v) { z[L::ix(e)] = v; });
    __syncthreads();
    if (!active) return;
    constexpr int nxh = L::N / 2 + 1;
    Cx<T> *ha = reinterpret_cast<Cx<T> *>(H) + (size_t)nxh * ((size_t)jj + (size_t)nrow_h * k), *hb = ha + nxh;
    for (int kx = t; kx < nxh; kx += L::G) {
        const Cx<T> zk = z[L::ix(kx)], zm = z[L::ix((L::N - kx) & (L::N - 1))];
        ha[kx] = Cx<T>{(zk.r + zm.r) * T(0.5), (zk.i - zm.i) * T(0.5)};
        hb[kx] = Cx<T>{(zk.i + zm.i) * T(0.5), (zm.r - zk.r) * T(0.5)};
    }
}

// row pairs per block of the register passes
inline int fft_reg_lines(int n, long lines) {
    int p = std::max(1, 2048 / n);
    while (p > 1 && p * n > 256 && (lines + p - 1) / p < FFT_MIN_BLOCKS) p >>= 1;
    return p;
}

template <typename T, typename TS>
inline void fft_x_fwd(int nb, Batch<const TS *> src, T *H, size_t hstride, int n, int nrow_src, int j0, int nrow_h,
                      int npairs, int nplanes, const T *twr, const T *twi, cudaStream_t s) {
    const long lines = (long)npairs * nplanes;
    if (fft_in_registers<T>(n, lines * nb)) {
        const int pl = fft_reg_lines(n, lines * nb);
        fft_by_length(n, [&](auto lg) {
            using L = LineFft<decltype(lg)::value>;
            k_fft_x_fwd_r<decltype(lg)::value, T, TS>
                <<<dim3((unsigned)((lines + pl - 1) / pl), 1, nb), pl * L::G, pl * L::PITCH * sizeof(Cx<T>), s>>>(
                    src, H, hstride, nrow_src, j0, nrow_h, npairs, nplanes, twr, twi);
        });
        count_launch();
        return;
    }
    const int ppc = fft_pairs_per_block(n, (long)npairs * nplanes * nb);
    const size_t smem = (size_t)ppc * 2 * n * sizeof(Cx<T>);
    const dim3 grid((unsigned)(((long)npairs * nplanes + ppc - 1) / ppc), 1, nb);
    k_fft_x_fwd<T, TS><<<grid, ppc * (n / 2), smem, s>>>(src, H, hstride, ilog2_pow2(n), nrow_src, j0, nrow_h, npairs,
                                                         nplanes, twr, twi);
    count_launch();
}

// Destinations of an inverse x pass.  XOutD: an FP64 field (FP64 path and
// stand-alone solve).  XOutF: the FP32 / double-float fields of the mixed path
// (modes below).
struct XOutD {
    double *dst;
    __device__ __forceinline__ void put(size_t o, double v) const { dst[o] = v; }
};

struct XOutF {
    float *hi, *lo;
    int mode;
    // mode 0: hi = v.  mode 2: (hi, lo) = hi + v exactly (two-sum), the
    // correction of an FP32 field to a df64 pair
    __device__ __forceinline__ void put(size_t o, float v) const {
        if (mode == 0) {
            hi[o] = v;
        } else {
            float s, e;
            two_sum(hi[o], v, s, e);
            hi[o] = s;
            lo[o] = e;
        }
    }
};

// Inverse: spectral rows jj, jj+1 (nrow_h per plane) -> real rows jdst0 + jj,
// jdst0 + jj + 1 of a halo-layout field (x written at 1..n) through the
// destination functor.
template <typename T, typename Out>
__global__ void k_fft_x_inv(const T *__restrict__ H, size_t hstride, Batch<Out> outs, int lg, int nrow_h,
                            int npairs_per_plane, int nplanes, int jdst0, int sx, int sy, const T *__restrict__ twr,
                            const T *__restrict__ twi, int plain) {
    extern __shared__ unsigned char smem_raw[];
    Cx<T> *sm = reinterpret_cast<Cx<T> *>(smem_raw);
    const int n = 1 << lg, half = n >> 1, tpp = half;
    const Out out = outs.p[blockIdx.z];
    H += (size_t)blockIdx.z * hstride;
    const int p = threadIdx.x >> (lg - 1), t = threadIdx.x & (half - 1);
    const long pair = (long)blockIdx.x * (blockDim.x >> (lg - 1)) + p;
    const bool active = pair < (long)npairs_per_plane * nplanes;
    Cx<T> *x = sm + (size_t)p * 2 * n, *y = x + n;
    int k = 0, jj = 0;
    const int nxh = half + 1;
    if (active) {
        k = (int)(pair / npairs_per_plane);
        jj = 2 * (int)(pair % npairs_per_plane);
        const T *ha = H + 2 * ((size_t)nxh * ((size_t)jj + (size_t)nrow_h * k));
        const T *hb = ha + 2 * nxh;
        for (int e = t; e < n; e += tpp) {
            if (e <= half) {
                T ar = ha[2 * e], ai = ha[2 * e + 1], br = hb[2 * e], bi = hb[2 * e + 1];
                x[e].r = ar - bi; x[e].i = ai + br;
            } else {
                int m = n - e;
                T ar = ha[2 * m], ai = ha[2 * m + 1], br = hb[2 * m], bi = hb[2 * m + 1];
                x[e].r = ar + bi; x[e].i = br - ai;
            }
        }
    }
    __syncthreads();
    for (int ls = 0; ls < lg; ++ls) {
        if (active) stockham_stage<true>(x, y, lg, ls, t, twr, twi, +1);
        __syncthreads();
        Cx<T> *tmp = x; x = y; y = tmp;
    }
    if (!active) return;
    // halo layout (x at 1..n) or, with plain, a dense [k][j][x] array of
    // row length n and sy rows per plane
    const size_t oa = plain ? (size_t)n * ((size_t)(jdst0 + jj) + (size_t)sy * k)
                            : 1 + (size_t)sx * ((size_t)(jdst0 + jj) + (size_t)sy * (k + 1));
    const size_t ob = oa + (plain ? n : sx);
    for (int e = t; e < n; e += tpp) { out.put(oa + e, x[e].r); out.put(ob + e, x[e].i); }
}

template <int LG, typename T, typename Out>
__global__ void __launch_bounds__(256) k_fft_x_inv_r(const T *__restrict__ H, size_t hstride, Batch<Out> outs, int nrow_h,
                                                     int npairs_per_plane, int nplanes, int jdst0, int sx, int sy,
                                                     const T *__restrict__ twr, const T *__restrict__ twi, int plain) {
    using L = LineFft<LG>;
    extern __shared__ unsigned char smem_raw[];
    const Out out = outs.p[blockIdx.z];
    H += (size_t)blockIdx.z * hstride;
    const int p = threadIdx.x / L::G, t = threadIdx.x % L::G;
    const long pair = (long)blockIdx.x * (blockDim.x / L::G) + p;
    const bool active = pair < (long)npairs_per_plane * nplanes;
    Cx<T> *z = reinterpret_cast<Cx<T> *>(smem_raw) + p * L::PITCH;
    const int k = active ? (int)(pair / npairs_per_plane) : 0, jj = active ? 2 * (int)(pair % npairs_per_plane) : 0;
    constexpr int half = L::N / 2, nxh = half + 1;
    const Cx<T> *ha = reinterpret_cast<const Cx<T> *>(H) + (size_t)nxh * ((size_t)jj + (size_t)nrow_h * k), *hb = ha + nxh;
    const size_t oa = plain ? (size_t)L::N * ((size_t)(jdst0 + jj) + (size_t)sy * k)
                            : 1 + (size_t)sx * ((size_t)(jdst0 + jj) + (size_t)sy * (k + 1));
    const size_t ob = oa + (plain ? L::N : sx);
    fft_line<true, LG, T>(
        z, t, twr, twi,
        [&](int e) {
            if (!active) return Cx<T>{T(0), T(0)};
            const int m = e <= half ? e : L::N - e;
            const Cx<T> a = ha[m], b = hb[m];
            return e <= half ? Cx<T>{a.r - b.i, a.i + b.r} : Cx<T>{a.r + b.i, b.r - a.i};
        },
        [&](int e, Cx<T> v) {
            if (!active) return;
            out.put(oa + e, v.r);
            out.put(ob + e, v.i);
        });
}

template <typename T, typename Out>
inline void fft_x_inv(int nb, const T *H, size_t hstride, Batch<Out> out, int n, int nrow_h, int npairs, int nplanes,
                      int jdst0, int sx, int sy, const T *twr, const T *twi, int plain, cudaStream_t s) {
    const long lines = (long)npairs * nplanes;
    if (fft_in_registers<T>(n, lines * nb)) {
        const int pl = fft_reg_lines(n, lines * nb);
        fft_by_length(n, [&](auto lg) {
            using L = LineFft<decltype(lg)::value>;
            k_fft_x_inv_r<decltype(lg)::value, T, Out>
                <<<dim3((unsigned)((lines + pl - 1) / pl), 1, nb), pl * L::G, pl * L::PITCH * sizeof(Cx<T>), s>>>(
                    H, hstride, out, nrow_h, npairs, nplanes, jdst0, sx, sy, twr, twi, plain);
        });
        count_launch();
        return;
    }
    const int ppc = fft_pairs_per_block(n, (long)npairs * nplanes * nb);
    const size_t smem = (size_t)ppc * 2 * n * sizeof(Cx<T>);
    const dim3 grid((unsigned)(((long)npairs * nplanes + ppc - 1) / ppc), 1, nb);
    k_fft_x_inv<T, Out><<<grid, ppc * (n / 2), smem, s>>>(H, hstride, out, ilog2_pow2(n), nrow_h, npairs, nplanes, jdst0,
                                                          sx, sy, twr, twi, plain);
    count_launch();
}

// ---------------------------------------------------------------------------
// Strided complex transforms along y or z of the half spectrum.  A CTA owns tx
// consecutive kx columns of one line set and keeps [tx][n] complex values in
// shared memory (so global reads are row segments of tx complex values).
//   line element e of column c: H[base + e*lstride + c]  (complex units)
//   base = set*sstride + kx0
// mode 0: single transform with sign; mode 1: forward, spectral divide,
// inverse (periodic solve, fenep.f90:1408-1426); the divide needs the
// modified-wavenumber tables and the line index of the other axes.
struct DivideSpec {
    const double *kx2, *ky2, *kz2;  // tables (FP64)
    double lhs0, lhs1;              // LHS = lhs0 + lhs1*((kx2+ky2)+kz2); Q/ntot/LHS
    double inv_ntot;                // 1/(nx ny nz), a power of two: the product is the quotient
    int line_is_z;                  // 1: line along z (set = j); 0: along y (set = k)
};

template <typename T>
__global__ void __launch_bounds__(256) k_fft_lines(T *__restrict__ H, size_t hstride, int lg, int lstride, int ncols,
                                                   int sstride, int tx, const T *__restrict__ twr,
                                                   const T *__restrict__ twi, int sign, int mode, DivideSpec dv) {
    extern __shared__ unsigned char smem_raw[];
    const int n = 1 << lg;
    Cx<T> *bufA = reinterpret_cast<Cx<T> *>(smem_raw);
    Cx<T> *bufB = bufA + (size_t)n * tx;
    const int set = blockIdx.y;
    const int kx0 = blockIdx.x * tx;
    const int ncol = min(tx, ncols - kx0);
    const int ltx = 31 - __clz(tx);     // tx is a power of two
    Cx<T> *Hc = reinterpret_cast<Cx<T> *>(H + (size_t)blockIdx.z * hstride);
    const size_t base = (size_t)set * sstride + kx0;
    // load: element (e, c) -> buf[c*n + e]
    for (int q = threadIdx.x; q < n * tx; q += blockDim.x) {
        const int e = q >> ltx, c = q & (tx - 1);
        if (c < ncol) bufA[(c << lg) + e] = Hc[base + (size_t)e * lstride + c];
    }
    __syncthreads();
    const int nbfly = ncol << (lg - 1);
    const int passes = mode == 1 ? 2 : 1;
    Cx<T> *x = bufA, *y = bufB;
    for (int ps = 0; ps < passes; ++ps) {
        const int sg = mode == 1 ? (ps == 0 ? -1 : +1) : sign;
        for (int ls = 0; ls < lg; ++ls) {
            for (int q = threadIdx.x; q < nbfly; q += blockDim.x) {
                const int c = q >> (lg - 1), j = q & ((n >> 1) - 1);
                if (sg < 0) stockham_stage<false>(x + (c << lg), y + (c << lg), lg, ls, j, twr, twi, sg);
                else stockham_stage<true>(x + (c << lg), y + (c << lg), lg, ls, j, twr, twi, sg);
            }
            __syncthreads();
            Cx<T> *tmp = x; x = y; y = tmp;
        }
        if (mode == 1 && ps == 0) {
            for (int q = threadIdx.x; q < ncol << lg; q += blockDim.x) {
                const int c = q >> lg, e = q & (n - 1);
                // element e of the line: along z -> kz = e, ky = set; along y -> ky = e, kz = set
                const int jy = dv.line_is_z ? set : e;
                const int kz = dv.line_is_z ? e : set;
                const double lhs = dv.lhs0 + dv.lhs1 * (dv.kx2[kx0 + c] + dv.ky2[jy] + dv.kz2[kz]);
                Cx<T> v = x[q];
                const T qr = v.r * T(dv.inv_ntot), qi = v.i * T(dv.inv_ntot);
                if (fabs(lhs) < 1.0e-16) { v.r = T(0); v.i = T(0); }
                else { v.r = qr / T(lhs); v.i = qi / T(lhs); }
                x[q] = v;
            }
            __syncthreads();
        }
    }
    for (int q = threadIdx.x; q < n * tx; q += blockDim.x) {
        const int e = q >> ltx, c = q & (tx - 1);
        if (c < ncol) Hc[base + (size_t)e * lstride + c] = x[(c << lg) + e];
    }
}

// mode 0 (INV: the sign) and 1 of k_fft_lines on register lines; neighbouring
// threads take neighbouring columns
template <int LG, bool SOLVE, bool INV, typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256)
k_fft_lines_r(T *__restrict__ H, size_t hstride, int lstride, int ncols, int sstride, int tx, const T *__restrict__ twr,
              const T *__restrict__ twi, DivideSpec dv) {
    using L = LineFft<LG>;
    extern __shared__ unsigned char smem_raw[];
    const int c = threadIdx.x & (tx - 1), t = threadIdx.x >> (31 - __clz(tx)), kx = blockIdx.x * tx + c, set = blockIdx.y;
    const bool active = kx < ncols;
    Cx<T> *z = reinterpret_cast<Cx<T> *>(smem_raw) + c * L::PITCH;
    Cx<T> *Hc = reinterpret_cast<Cx<T> *>(H + (size_t)blockIdx.z * hstride) + (size_t)set * sstride + kx;
    auto load = [&](int e) { return active ? Hc[(size_t)e * lstride] : Cx<T>{T(0), T(0)}; };
    auto store = [&](int e, Cx<T> v) {
        if (active) Hc[(size_t)e * lstride] = v;
    };
    if constexpr (!SOLVE) {
        fft_line<INV, LG, T>(z, t, twr, twi, load, store);
    } else {
        Cx<T> keep[8];
        int at = 0;
        fft_line<false, LG, T>(z, t, twr, twi, load, [&](int e, Cx<T> v) {
            // element e of the line: along z -> kz = e, ky = set; along y -> ky = e, kz = set
            const int jy = dv.line_is_z ? set : e, kz = dv.line_is_z ? e : set;
            const double lhs = dv.lhs0 + dv.lhs1 * (dv.kx2[active ? kx : 0] + dv.ky2[jy] + dv.kz2[kz]);
            const T qr = v.r * T(dv.inv_ntot), qi = v.i * T(dv.inv_ntot);
            keep[at++] = fabs(lhs) < 1.0e-16 ? Cx<T>{T(0), T(0)} : Cx<T>{qr / T(lhs), qi / T(lhs)};
        });
        __syncthreads();      // the last pass has read the line
        constexpr int RL = LG == 5 || LG == 7 || LG == 8 || LG == 10 ? 2 : 3, L0 = LG - RL, W = 1 << RL;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int g = t + q / W * L::G, e = ((g >> L0) << LG) | (g & ((1 << L0) - 1)) | (q % W << L0);
            z[L::ix(e)] = keep[q];
        }
        __syncthreads();
        Cx<T> in[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) in[s] = z[L::ix(L::brev(8 * t + s))];
        __syncthreads();
        at = 0;
        fft_line<true, LG, T>(z, t, twr, twi, [&](int) { return in[at++]; }, store);
    }
}

template <typename T>
inline void fft_lines(int nb, T *H, size_t hstride, int n, int lstride, int ncols, int sets, int sstride, const T *twr,
                      const T *twi, int sign, int mode, const DivideSpec &dv, cudaStream_t s) {
    const int tx = fft_cols_per_block<T>(n, ncols, (long)sets * nb);
    if (fft_in_registers<T>(n, (long)ncols * sets * nb)) {
        fft_by_length(n, [&](auto lg) {
            constexpr int LG = decltype(lg)::value;
            using L = LineFft<LG>;
            auto go = [&](auto kernel) {
                kernel<<<dim3((ncols + tx - 1) / tx, sets, nb), tx * L::G, tx * L::PITCH * sizeof(Cx<T>), s>>>(
                    H, hstride, lstride, ncols, sstride, tx, twr, twi, dv);
            };
            if (mode == 1) go(k_fft_lines_r<LG, true, false, T>);
            else if (sign < 0) go(k_fft_lines_r<LG, false, false, T>);
            else go(k_fft_lines_r<LG, false, true, T>);
        });
        count_launch();
        return;
    }
    const size_t smem = (size_t)2 * n * tx * sizeof(Cx<T>);
    k_fft_lines<T><<<dim3((ncols + tx - 1) / tx, sets, nb), fft_line_threads<T>(n, tx), smem, s>>>(
        H, hstride, ilog2_pow2(n), lstride, ncols, sstride, tx, twr, twi, sign, mode, dv);
    count_launch();
}

// The periodic solve (fft_solve, fenep.f90:1400-1428) of nb right-hand sides
// (interior order) through their spectra H: five passes in 3D; in 2D (nz = 1)
// the y lines transform, divide and transform back in one of three.
template <typename T, typename TS, typename Out>
inline void fft_solve_passes(int nb, Batch<const TS *> src, T *H, size_t hstride, Batch<Out> out, int nx, int ny, int nz,
                             int jdst0, int sx, int sy, int plain, const T *twx_r, const T *twx_i, const T *twy_r,
                             const T *twy_i, const T *twz_r, const T *twz_i, const double *kx2, const double *ky2,
                             const double *kz2, double lhs0, double lhs1, cudaStream_t s) {
    const int nxh = nx / 2 + 1;
    const DivideSpec dv{kx2, ky2, kz2, lhs0, lhs1, 1.0 / ((double)nx * ny * nz), nz > 1 ? 1 : 0};
    fft_x_fwd<T, TS>(nb, src, H, hstride, nx, ny, 1, ny, ny / 2, nz, twx_r, twx_i, s);
    if (nz == 1) {
        fft_lines<T>(nb, H, hstride, ny, nxh, nxh, 1, nxh * ny, twy_r, twy_i, -1, 1, dv, s);
    } else {
        fft_lines<T>(nb, H, hstride, ny, nxh, nxh, nz, nxh * ny, twy_r, twy_i, -1, 0, dv, s);
        fft_lines<T>(nb, H, hstride, nz, nxh * ny, nxh, ny, nxh, twz_r, twz_i, -1, 1, dv, s);
        fft_lines<T>(nb, H, hstride, ny, nxh, nxh, nz, nxh * ny, twy_r, twy_i, +1, 0, dv, s);
    }
    fft_x_inv<T, Out>(nb, H, hstride, out, nx, ny, ny / 2, nz, jdst0, sx, sy, twx_r, twx_i, plain, s);
}

// ---------------------------------------------------------------------------
// Wall-normal systems (fenep_2d.f90:1222-1238, 1262-1277, 1318-1332 with
// NA = 0, NB = NY; x and z periodic): rows j = 0..NY+1 of the spectrum, the
// right-hand side in rows 1..NY, the Thomas recurrence of tdma with the
// reference's near-zero-pivot guard.
enum WallSys { SYS_U = 0, SYS_V = 1, SYS_P = 2 };

struct WallSpec {
    const double *kx2, *kz2;
    double dt, beta, re, dy;
    double nxz;     // NX*NZ normalisation of the forward transforms
};

inline WallSpec wall_spec(const Geo &g, const Phys &ph, const double *kx2, const double *kz2) {
    return WallSpec{kx2, kz2, ph.dt, ph.beta, ph.re, g.dy, (double)g.nx * g.nz};
}

// One system of a batched wall solve: the tables of its kind, and the value of
// the top ghost row of mode (0, 0) (2*uwall for U)
template <typename T>
struct WallItem {
    int sys;
    const T *tab;
    double top;
};

template <typename T>
__host__ __device__ inline void wall_coef(const WallSpec &w, int sys, int j, int ny, double lam, T &a, T &b, T &c) {
    const int n = ny + 2;
    if (sys == SYS_U) {
        if (j == 0) { a = T(1.0); b = T(1.0); c = T(0.0); }
        else if (j == n - 1) { a = T(1.0); b = T(0.0); c = T(1.0); }
        else {
            a = T(1.0 + w.dt * w.beta / w.re / 2.0 * (lam + 2.0 / (w.dy * w.dy)));
            b = T(-w.dt * w.beta / w.re / 2.0 / (w.dy * w.dy));
            c = b;
        }
    } else if (sys == SYS_V) {
        if (j == 0 || j >= ny) { a = T(1.0); b = T(0.0); c = T(0.0); }
        else {
            a = T(1.0 + w.dt * w.beta / w.re / 2.0 * (lam + 2.0 / (w.dy * w.dy)));
            b = T(-w.dt * w.beta / w.re / 2.0 / (w.dy * w.dy));
            c = b;
        }
    } else {
        if (j == 0) { a = T(1.0); b = T(-1.0); c = T(0.0); }
        else if (j == n - 1) { a = T(1.0); b = T(0.0); c = T(-1.0); }
        else {
            a = T(-(lam + 2.0 / (w.dy * w.dy)));
            b = T(1.0 / (w.dy * w.dy));
            c = b;
        }
    }
}

// Tables of the Thomas recurrence of every (kx, kz) system: per row and mode
// P = -b/den and den, in FP64 1/den as the sum of two doubles (f8_recip.cuh) in
// the second and third table, in FP32 den itself (an FP32 division is cheap).
// Where tdma's guard sets P = Q = 0 (fenep_2d.f90:1157-1160): P = 1/den = 0,
// den = inf.  Layout [row][kz][kx].
template <typename T>
__global__ void k_wall_table(T *__restrict__ P, T *__restrict__ rh, T *__restrict__ rl, int ny, int nxh, int nz,
                             WallSpec w, int sys) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nxh * nz) return;
    const double lam = w.kx2[q % nxh] + w.kz2[q / nxh];
    T p = T(0);
    for (int j = 0; j < ny + 2; ++j) {
        T a, b, cc;
        wall_coef<T>(w, sys, j, ny, lam, a, b, cc);
        const T den = j == 0 ? a : a + cc * p;
        const size_t o = (size_t)j * nxh * nz + q;
        const bool guard = j > 0 && fabs(den) < T(1.0e-16);
        p = guard ? T(0) : -b / den;
        P[o] = p;
        if constexpr (sizeof(T) == 8) {
            const Recip r = guard ? Recip{0.0, 0.0} : recip(den);
            rh[o] = r.h;
            rl[o] = r.l;
        } else {
            rh[o] = guard ? __int_as_float(0x7f800000) : den;
        }
    }
}

// t / den with those tables
__device__ __forceinline__ double wall_div(double t, double h, double l) { return div_by(t, Recip{h, l}); }
__device__ __forceinline__ float wall_div(float t, float den, float) { return t / den; }

// The wall-normal solves (tdma, fenep_2d.f90:1145-1177) of every mode with
// those tables.  A thread runs the recurrence of the real or the imaginary part
// of one mode (the coefficients are real), neighbouring threads neighbouring
// values of a row, so the rows stream through without a tile; the forward
// values wait in the rows of the right-hand side.  In FP64 the chain is 5 slots a
// row forward and 2 back, where forming the coefficients and dividing took about 60 in a
// half-filled warp.
template <typename T>
__global__ void __launch_bounds__(64) k_wall_tdma(T *H, size_t hstride, int ny, int nxh, int nz, T inv_nxz,
                                                  Batch<WallItem<T>> items, Batch<T> off) {
    const int n = ny + 2;
    const WallItem<T> it = items.p[blockIdx.z];
    const int sys = it.sys;
    const T ci = off.p[blockIdx.z];                         // the interior rows' off-diagonal
    const size_t modes = (size_t)nxh * nz;
    const T *__restrict__ P = it.tab, *__restrict__ rh = P + modes * n, *__restrict__ rl = rh + modes * n;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;   // kx * 2 + part
    const int kz = blockIdx.y;
    if (c >= 2 * nxh) return;
    const size_t mode = (size_t)nxh * kz + (c >> 1);
    T *h0 = H + blockIdx.z * hstride + (size_t)2 * nxh * n * kz + c;
    T q = T(0);
    // in groups of 8 rows: the loads do not depend on the recurrence, so a group's
    // are all in flight before its chain begins
    constexpr int G = 8;
    for (int j0 = 0; j0 < n; j0 += G) {
        T d[G], h[G], l[G];
#pragma unroll
        for (int u = 0; u < G; ++u) {
            const int j = j0 + u;
            d[u] = h[u] = l[u] = T(0);
            if (j >= n) continue;
            if (j >= 1 && j <= ny && !(sys == SYS_V && j == ny)) d[u] = h0[(size_t)2 * nxh * j] * inv_nxz;
            else if (j == n - 1 && mode == 0 && c == 0) d[u] = T(it.top);
            h[u] = rh[(size_t)j * modes + mode];
            if (sizeof(T) == 8) l[u] = rl[(size_t)j * modes + mode];
        }
#pragma unroll
        for (int u = 0; u < G; ++u) {
            const int j = j0 + u;
            if (j >= n) continue;
            const T cc = j == 0 ? T(0) : (j == n - 1 ? (sys == SYS_U ? T(1) : (sys == SYS_V ? T(0) : T(-1)))
                                                     : (sys == SYS_V && j >= ny ? T(0) : ci));
            const T t = d[u] - cc * q;
            q = wall_div(t, h[u], l[u]);
            h0[(size_t)2 * nxh * j] = q;
        }
    }
    T x = q;
    for (int j0 = n - 2; j0 >= 0; j0 -= G) {
        T p[G], r[G];
#pragma unroll
        for (int u = 0; u < G; ++u) {
            const int j = j0 - u;
            p[u] = r[u] = T(0);
            if (j < 0) continue;
            p[u] = P[(size_t)j * modes + mode];
            r[u] = h0[(size_t)2 * nxh * j];
        }
#pragma unroll
        for (int u = 0; u < G; ++u) {
            const int j = j0 - u;
            if (j < 0) continue;
            x = p[u] * x + r[u];
            h0[(size_t)2 * nxh * j] = x;
        }
    }
}

template <typename T>
inline void wall_table(T *tab, int ny, int nxh, int nz, const WallSpec &w, int sys, cudaStream_t s) {
    const size_t m = (size_t)(ny + 2) * nxh * nz;
    k_wall_table<T><<<(nxh * nz + 127) / 128, 128, 0, s>>>(tab, tab + m, tab + 2 * m, ny, nxh, nz, w, sys);
    count_launch();
}

template <typename T>
inline void wall_tdma(int nb, T *H, size_t hstride, int ny, int nxh, int nz, const WallSpec &w,
                      Batch<WallItem<T>> items, cudaStream_t s) {
    Batch<T> off{};
    for (int q = 0; q < nb; ++q) {
        T a, b;
        wall_coef<T>(w, items.p[q].sys, 1, ny, 0.0, a, b, off.p[q]);
    }
    k_wall_tdma<T><<<dim3((2 * nxh + 63) / 64, nz, nb), 64, 0, s>>>(H, hstride, ny, nxh, nz, T(1.0 / w.nxz), items, off);
    count_launch();
}

// The wall-bounded solves of nb systems: FFT(x, z) of rows 1..NY, the
// tridiagonal systems in y over rows 0..NY+1, inverse FFT of all NY+2 rows into
// the halo rows of out.  H holds nb spectra of ny + 2 rows.
template <typename T, typename TS, typename Out>
inline void wall_solve_passes(int nb, Batch<const TS *> src, T *H, size_t hstride, Batch<Out> out, const Geo &g,
                              const T *twx_r, const T *twx_i, const T *twz_r, const T *twz_i, const WallSpec &w,
                              Batch<WallItem<T>> items, cudaStream_t s) {
    const int nx = g.nx, ny = g.ny, nz = g.nz, nxh = nx / 2 + 1, n = ny + 2;
    const DivideSpec none{};
    T *H1 = H + (size_t)2 * nxh;      // row 1
    fft_x_fwd<T, TS>(nb, src, H1, hstride, nx, ny, 1, n, ny / 2, nz, twx_r, twx_i, s);
    if (nz > 1) fft_lines<T>(nb, H1, hstride, nz, nxh * n, nxh, ny, nxh, twz_r, twz_i, -1, 0, none, s);
    wall_tdma<T>(nb, H, hstride, ny, nxh, nz, w, items, s);
    if (nz > 1) fft_lines<T>(nb, H, hstride, nz, nxh * n, nxh, n, nxh, twz_r, twz_i, +1, 0, none, s);
    fft_x_inv<T, Out>(nb, H, hstride, out, nx, n, n / 2, nz, 0, g.sx, g.sy, twx_r, twx_i, 0, s);
}

}  // namespace f8
