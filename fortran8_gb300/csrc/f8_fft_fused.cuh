// f8_fft_fused.cuh — FP32 spectral solves of the mixed-precision path with the
// whole (z, y) plane of one x-wavenumber resident in shared memory.
//
// Spectrum layout S[kx][k][j] (complex float), j contiguous, LJ values per
// (kx, k) line: LJ = NY for periodic y, NY + 2 for walls (rows 0 and NY+1 are
// the ghost rows of the wall systems, fenep_2d.f90:1222-1238).
//
//   k_xfwd_t   real rows -> S: two rows per complex FFT of length NX (the
//              same pairing as the FP64 kernels), transposed through shared
//              memory so that each kx receives RB consecutive rows.
//   k_xfwd_w, k_xinv_w   the x passes of NX = 32 .. 512 in registers
//   k_plane_*  one CTA (or a cluster) per kx: transforms along z (and y
//              when periodic), the spectral divide (fft_solve, fenep.f90:1400-
//              1428) or the Thomas solve along y (tdma, fenep_2d.f90:1145-1177),
//              and the inverse transforms.  Forward transforms leave their
//              values in bit-reversed order, inverse ones take them so.
//   k_xinv_t   S -> real rows through a destination functor (XOutF).
#pragma once
#include <cooperative_groups.h>
#include "f8_common.cuh"
#include "f8_fft.cuh"

namespace f8 {

__device__ inline int bitrev(int v, int lg) { return lg ? (int)(__brev((unsigned)v) >> (32 - lg)) : 0; }

// a * w: (fma(ax, wx, -(ay wy)), fma(ax, wy, ay wx)).  Four scalar operations:
// the packed FP32x2 form of the same bits is two, but needs (ax, ax), (ay, ay)
// and (-wy, wx) in register pairs, four moves on the same issue slots.
__device__ __forceinline__ float2 cmul_p(float2 a, float2 w) {
    return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}

// ---------------------------------------------------------------------------
// x forward, transposing.  Block b handles RB rows (RB/2 pairs) of plane k.
// The [kx][row] tile has an odd row stride (RB + 1) against bank conflicts.
template <typename TS>
__global__ void k_xfwd_t(const TS *__restrict__ src, float2 *__restrict__ S, int nx, int ny, int nz, int rb, int lj,
                         int joff, const float *__restrict__ twr, const float *__restrict__ twi) {
    extern __shared__ unsigned char smem_raw[];
    Cx<float> *sm = reinterpret_cast<Cx<float> *>(smem_raw);
    const int half = nx >> 1, nxh = half + 1;
    const int npair = rb >> 1;
    const int p = threadIdx.x / half, t = threadIdx.x % half;
    const int blocks_per_plane = (ny + rb - 1) / rb;
    const int k = blockIdx.x / blocks_per_plane;
    const int r0 = (blockIdx.x % blocks_per_plane) * rb;       // first row (0-based) of the block
    const int nrows = min(rb, ny - r0);
    const bool active = p < npair && 2 * p < nrows;
    Cx<float> *x = sm + (size_t)p * 2 * nx, *y = x + nx;
    if (active) {
        const TS *ra = src + (size_t)nx * ((size_t)(r0 + 2 * p) + (size_t)ny * k);
        const TS *rbp = ra + nx;
        for (int e = t; e < nx; e += half) { x[e].r = (float)ra[e]; x[e].i = (float)rbp[e]; }
    }
    __syncthreads();
    const int lg = ilog2_pow2(nx);
    for (int ls = 0; ls < lg; ++ls) {
        if (active) stockham_stage<false>(x, y, lg, ls, t, twr, twi, -1);
        __syncthreads();
        Cx<float> *tmp = x; x = y; y = tmp;
    }
    // unpack the two real spectra of each pair into a [kx][row] tile; the
    // result of pair p is in buffer x (the same buffer index for all pairs)
    const bool res_in_first = ((__ffs(nx) - 1) % 2) == 0;  // log2(nx) even -> back in the first buffer
    float2 *tile = reinterpret_cast<float2 *>(sm + (size_t)npair * 2 * nx);
    if (active) {
        const Cx<float> *z = sm + (size_t)p * 2 * nx + (res_in_first ? 0 : nx);
        for (int kx = t; kx < nxh; kx += half) {
            const int m = (nx - kx) % nx;
            const Cx<float> zk = z[kx], zm = z[m];
            tile[(size_t)kx * (rb + 1) + 2 * p] = make_float2((zk.r + zm.r) * 0.5f, (zk.i - zm.i) * 0.5f);
            tile[(size_t)kx * (rb + 1) + 2 * p + 1] = make_float2((zk.i + zm.i) * 0.5f, (zm.r - zk.r) * 0.5f);
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nxh * rb; q += blockDim.x) {
        const int kx = q / rb, r = q % rb;
        if (r < nrows) S[((size_t)kx * nz + k) * lj + (r0 + r + 1 + joff)] = tile[(size_t)kx * (rb + 1) + r];
    }
}

// x inverse, transposing: rows j = jlo .. jlo+nrow-1 of S (S row index
// j + joff2) become real rows j of a halo-layout field (x at 1..nx), written
// through the destination functor (XOutF).
template <typename Out>
__global__ void k_xinv_t(const float2 *__restrict__ S, Out out, int nx, int nrow, int jlo, int nz,
                         int rb, int lj, int joff2, int sx, int sy, const float *__restrict__ twr,
                         const float *__restrict__ twi) {
    extern __shared__ unsigned char smem_raw[];
    Cx<float> *sm = reinterpret_cast<Cx<float> *>(smem_raw);
    const int half = nx >> 1, nxh = half + 1;
    const int npair = rb >> 1;
    const int blocks_per_plane = (nrow + rb - 1) / rb;
    const int k = blockIdx.x / blocks_per_plane;
    const int r0 = (blockIdx.x % blocks_per_plane) * rb;
    const int nrows = min(rb, nrow - r0);
    float2 *tile = reinterpret_cast<float2 *>(sm + (size_t)npair * 2 * nx);
    for (int q = threadIdx.x; q < nxh * rb; q += blockDim.x) {
        const int kx = q / rb, r = q % rb;
        tile[(size_t)kx * (rb + 1) + r] = r < nrows ? S[((size_t)kx * nz + k) * lj + (jlo + r0 + r + joff2)] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int p = threadIdx.x / half, t = threadIdx.x % half;
    const bool active = p < npair && 2 * p < nrows;
    Cx<float> *x = sm + (size_t)p * 2 * nx, *y = x + nx;
    if (active) {
        for (int e = t; e < nx; e += half) {
            float ar, ai, br, bi;
            if (e <= half) {
                const float2 A = tile[(size_t)e * (rb + 1) + 2 * p], B = tile[(size_t)e * (rb + 1) + 2 * p + 1];
                ar = A.x; ai = A.y; br = B.x; bi = B.y;
                x[e].r = ar - bi; x[e].i = ai + br;
            } else {
                const int m = nx - e;
                const float2 A = tile[(size_t)m * (rb + 1) + 2 * p], B = tile[(size_t)m * (rb + 1) + 2 * p + 1];
                ar = A.x; ai = A.y; br = B.x; bi = B.y;
                x[e].r = ar + bi; x[e].i = br - ai;
            }
        }
    }
    __syncthreads();
    const int lg = ilog2_pow2(nx);
    for (int ls = 0; ls < lg; ++ls) {
        if (active) stockham_stage<true>(x, y, lg, ls, t, twr, twi, +1);
        __syncthreads();
        Cx<float> *tmp = x; x = y; y = tmp;
    }
    if (!active) return;
    const size_t oa = 1 + (size_t)sx * ((size_t)(jlo + r0 + 2 * p) + (size_t)sy * (k + 1));
    const bool has_b = 2 * p + 1 < nrows;
    for (int e = t; e < nx; e += half) {
        out.put(oa + e, x[e].r);
        if (has_b) out.put(oa + sx + e, x[e].i);
    }
}

// ---------------------------------------------------------------------------
// In-place radix-2 stages over nlines lines of length n held in shared memory
// (element e of line l at P[l*lstride_l + e*estride]).
__device__ inline void dit_lines(float2 *P, int n, int lg, int nlines, int lstride, int estride, const float *twr,
                                 const float *twi, float sign) {
    const int half = n >> 1;
    for (int m = 1; m < n; m <<= 1) {
        const int tws = n / (2 * m);
        for (int q = threadIdx.x; q < nlines * half; q += blockDim.x) {
            // consecutive threads take consecutive addresses: along the line
            // when it is contiguous, across lines otherwise
            const int l = estride == 1 ? q / half : q % nlines;
            const int b = estride == 1 ? q % half : q / nlines;
            const int pos = b % m, grp = b / m;
            const int i0 = grp * 2 * m + pos;
            float2 *base = P + (size_t)l * lstride;
            const float wr = twr[pos * tws], wi = sign * twi[pos * tws];
            const float2 a = base[(size_t)i0 * estride], c = base[(size_t)(i0 + m) * estride];
            const float tr = c.x * wr - c.y * wi, ti = c.x * wi + c.y * wr;
            base[(size_t)i0 * estride] = make_float2(a.x + tr, a.y + ti);
            base[(size_t)(i0 + m) * estride] = make_float2(a.x - tr, a.y - ti);
        }
        __syncthreads();
    }
    (void)lg;
}

__device__ inline void dif_lines(float2 *P, int n, int nlines, int lstride, int estride, const float *twr,
                                 const float *twi, float sign) {
    const int half = n >> 1;
    for (int m = half; m >= 1; m >>= 1) {
        const int tws = n / (2 * m);
        for (int q = threadIdx.x; q < nlines * half; q += blockDim.x) {
            const int l = estride == 1 ? q / half : q % nlines;
            const int b = estride == 1 ? q % half : q / nlines;
            const int pos = b % m, grp = b / m;
            const int i0 = grp * 2 * m + pos;
            float2 *base = P + (size_t)l * lstride;
            const float wr = twr[pos * tws], wi = sign * twi[pos * tws];
            const float2 a = base[(size_t)i0 * estride], c = base[(size_t)(i0 + m) * estride];
            const float dr = a.x - c.x, di = a.y - c.y;
            base[(size_t)i0 * estride] = make_float2(a.x + c.x, a.y + c.y);
            base[(size_t)(i0 + m) * estride] = make_float2(dr * wr - di * wi, dr * wi + di * wr);
        }
        __syncthreads();
    }
}

// Walls in y, general NZ: coefficients of the y systems
struct WallPlane {
    const float *kx2, *kz2;   // modified wavenumbers
    float ai_base, bc;        // interior a = ai_base + kap * lam; b = c = bc
    float kap;                // dt beta / (2 Re) (Helmholtz) or -1 (Poisson: a = -(lam + 2/dy^2))
    int sys;                  // WallSys
    float nxz_inv;            // 1 / (NX NZ)
};

// Walls in y: forward z transform of rows 1..NY, Thomas solve along y of each
// kz over rows 0..NY+1 with the boundary rows of the system (homogeneous:
// the mixed path solves for increments), inverse z transform of all rows.
__global__ void k_plane_walls(float2 *S, int ny, int nz, int lgz, const float *twzr, const float *twzi, WallPlane ps) {
    extern __shared__ unsigned char smem_raw[];
    const int lj = ny + 2;
    const int ljs = lj | 1;                                            // odd shared-memory row stride
    float2 *P = reinterpret_cast<float2 *>(smem_raw);                 // [k][j], k bit-reversed on load
    float *Pc = reinterpret_cast<float *>(P + (size_t)ljs * nz);      // Thomas P coefficients [k][j]
    const int kx = blockIdx.x;
    float2 *Sp = S + (size_t)kx * nz * lj;
    for (int q = threadIdx.x; q < lj * nz; q += blockDim.x) {
        const int k = q / lj, j = q % lj;
        P[(size_t)bitrev(k, lgz) * ljs + j] = (j >= 1 && j <= ny) ? Sp[q] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    dit_lines(P + 1, nz, lgz, ny, 1, ljs, twzr, twzi, 1.0f);  // lines j = 1..ny, along k
    // Thomas along j for each kz (natural order after DIT)
    const float lamx = ps.kx2[kx];
    for (int kz = threadIdx.x; kz < nz; kz += blockDim.x) {
        float2 *x = P + (size_t)kz * ljs;
        float *pc = Pc + (size_t)kz * ljs;
        const float lam = lamx + ps.kz2[kz];
        float ai, bc = ps.bc;
        if (ps.sys == SYS_P) ai = -(lam + ps.ai_base);
        else ai = ps.ai_base + ps.kap * lam;
        // row 0
        float a0, b0;
        if (ps.sys == SYS_U) { a0 = 1.f; b0 = 1.f; }
        else if (ps.sys == SYS_V) { a0 = 1.f; b0 = 0.f; }
        else { a0 = 1.f; b0 = -1.f; }
        float p = -b0 / a0;
        float2 qv = make_float2(0.f, 0.f);
        pc[0] = p; x[0] = qv;
        for (int j = 1; j < lj; ++j) {
            float a, b, c;
            float2 d;
            const bool last = j == lj - 1;
            if (ps.sys == SYS_U) {
                if (last) { a = 1.f; b = 0.f; c = 1.f; d = make_float2(0.f, 0.f); }
                else { a = ai; b = bc; c = bc; d = x[j]; d.x *= ps.nxz_inv; d.y *= ps.nxz_inv; }
            } else if (ps.sys == SYS_V) {
                if (j >= ny) { a = 1.f; b = 0.f; c = 0.f; d = make_float2(0.f, 0.f); }
                else { a = ai; b = bc; c = bc; d = x[j]; d.x *= ps.nxz_inv; d.y *= ps.nxz_inv; }
            } else {
                if (last) { a = 1.f; b = 0.f; c = -1.f; d = make_float2(0.f, 0.f); }
                else { a = ai; b = bc; c = bc; d = x[j]; d.x *= ps.nxz_inv; d.y *= ps.nxz_inv; }
            }
            // true divisions, as tdma does: on the singular Neumann mode of the
            // pressure system p stays exactly 1 and the last pivot is exactly
            // zero, so the reference's guard pins that mode
            const float den = a + c * p;
            if (fabsf(den) < 1.0e-16f) {
                p = 0.f; qv = make_float2(0.f, 0.f);
            } else {
                p = -b / den;
                qv = make_float2((d.x - c * qv.x) / den, (d.y - c * qv.y) / den);
            }
            pc[j] = p; x[j] = qv;
        }
        float2 xv = x[lj - 1];
        for (int j = lj - 2; j >= 0; --j) {
            const float pj = pc[j];
            const float2 qj = x[j];
            xv = make_float2(pj * xv.x + qj.x, pj * xv.y + qj.y);
            x[j] = xv;
        }
    }
    __syncthreads();
    dif_lines(P, nz, lj, 1, ljs, twzr, twzi, -1.0f);         // all rows, along k
    for (int q = threadIdx.x; q < lj * nz; q += blockDim.x) {
        const int k = q / lj, j = q % lj;
        Sp[q] = P[(size_t)bitrev(k, lgz) * ljs + j];
    }
}

// ---------------------------------------------------------------------------
// Radix-2 passes in registers over the V elements t + S s (s < V) of a line.
// tw: forward twiddles in shared memory, stage-major: the stage of span m
// reads w^(p N / (2m)), p < m, at tw[m - 1 + p], w = (cos, -sin)(2 pi / N), so
// that neighbouring t read consecutive entries.  With S = 1 the first twiddle
// of a stage is one.
//
// Forward, decimation in frequency, spans S V / 2 .. S (natural in, bit-reversed out)
template <int V, int S>
__device__ __forceinline__ void reg_dif(float2 (&v)[V], const float2 *tw, int t) {
#pragma unroll
    for (int m = V / 2; m >= 1; m >>= 1) {
        const float2 *tm = tw + (m * S - 1) + t;
#pragma unroll
        for (int p = 0; p < m; ++p) {
            const float2 w = S == 1 && p == 0 ? make_float2(1.0f, 0.0f) : tm[S * p];
#pragma unroll
            for (int s = p; s < V; s += 2 * m) {
                const float2 a = v[s], b = v[s + m];
                v[s] = __fadd2_rn(a, b);
                const float2 c = __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
                v[s + m] = S == 1 && p == 0 ? c : cmul_p(c, w);
            }
        }
    }
}

// Inverse (conjugate twiddles), decimation in time, spans S .. S V / 2
template <int V, int S>
__device__ __forceinline__ void reg_dit(float2 (&v)[V], const float2 *tw, int t) {
#pragma unroll
    for (int m = 1; m < V; m <<= 1) {
        const float2 *tm = tw + (m * S - 1) + t;
#pragma unroll
        for (int p = 0; p < m; ++p) {
            float2 w = S == 1 && p == 0 ? make_float2(1.0f, 0.0f) : tm[S * p];
            w.y = -w.y;
#pragma unroll
            for (int s = p; s < V; s += 2 * m) {
                const float2 a = v[s], c = S == 1 && p == 0 ? v[s + m] : cmul_p(v[s + m], w);
                v[s] = __fadd2_rn(a, c);
                v[s + m] = __ffma2_rn(c, make_float2(-1.0f, -1.0f), a);
            }
        }
    }
}

// Periodic y and z: the (z, y) plane of one kx is transformed, divided by
// ntot * LHS (LHS = lhs0 + lhs1 (kx2 + ky2 + kz2); zero where |LHS| < 1e-16) and
// transformed back.
struct PlaneSpec {
    const float *kx2, *ky2, *kz2;   // modified wavenumbers (FP32 copies)
    const float2 *twy, *twz;        // stage-major twiddles
    float lhs0, lhs1, inv_ntot;
};

// lanes per line, lines per warp and elements per lane of an N-point line (with
// N < 32 a warp holds 32 / N lines of N consecutive lanes)
template <int N>
struct LineOf {
    static constexpr int V = N >= 32 ? N / 32 : 1, L = N >= 32 ? 32 : N, W = 32 / L;
};
template <int N>
__device__ __forceinline__ int line_brev(int e) {
    constexpr int LG = N == 4 ? 2 : N == 8 ? 3 : N == 16 ? 4 : N == 32 ? 5 : N == 64 ? 6 : N == 128 ? 7 : N == 256 ? 8 : 9;
    return (int)(__brev((unsigned)e) >> (32 - LG));
}

// Forward transform, decimation in time: the value at position p of the line
// (lane p % 32, element p / 32) is that of index brev(p); out in natural order.
// In the butterflies a + b w, a - b w the lanes holding b multiply before the
// exchange.
template <int N>
__device__ __forceinline__ void line_dit_fwd(float2 (&v)[LineOf<N>::V], const float2 *tw, int lane) {
    constexpr int V = LineOf<N>::V;
#pragma unroll
    for (int m = 1; m < N; m <<= 1) {
        const float2 *tm = tw + (m - 1);
        if (m >= 32) {
            const int sm = m / 32;
#pragma unroll
            for (int s = 0; s < V; ++s) {
                if ((s / sm) % 2) continue;
                const float2 t = cmul_p(v[s + sm], tm[(lane + 32 * s) % (2 * m)]), a = v[s];
                v[s] = __fadd2_rn(a, t);
                v[s + sm] = make_float2(a.x - t.x, a.y - t.y);
            }
        } else {
            const bool second = lane & m;
            const float2 w = tm[lane & (m - 1)];
#pragma unroll
            for (int s = 0; s < V; ++s) {
                const float2 t = cmul_p(v[s], w);
                const float2 p = second ? t : v[s];
                const float ox = __shfl_xor_sync(0xffffffffu, p.x, m), oy = __shfl_xor_sync(0xffffffffu, p.y, m);
                v[s] = second ? make_float2(ox - p.x, oy - p.y) : make_float2(p.x + ox, p.y + oy);
            }
        }
    }
}

// d * conj(w) with the sum's fused product as twiddle_mul<true> has it
__device__ __forceinline__ float2 cmul_conj(float2 d, float2 w) {
    return __ffma2_rn(d, make_float2(w.x, w.x), __fmul2_rn(make_float2(d.y, d.x), make_float2(w.y, -w.y)));
}

// Inverse transform, decimation in frequency: natural order in, the value at
// position p is that of index brev(p)
template <int N>
__device__ __forceinline__ void line_dif_inv(float2 (&v)[LineOf<N>::V], const float2 *tw, int lane) {
    constexpr int V = LineOf<N>::V;
#pragma unroll
    for (int m = N / 2; m >= 1; m >>= 1) {
        const float2 *tm = tw + (m - 1);
        if (m >= 32) {
            const int sm = m / 32;
#pragma unroll
            for (int s = 0; s < V; ++s) {
                if ((s / sm) % 2) continue;
                const float2 a = v[s], b = v[s + sm];
                v[s] = __fadd2_rn(a, b);
                v[s + sm] = cmul_conj(make_float2(a.x - b.x, a.y - b.y), tm[(lane + 32 * s) % (2 * m)]);
            }
        } else {
            const bool second = lane & m;
            const float2 w = tm[lane & (m - 1)];
#pragma unroll
            for (int s = 0; s < V; ++s) {
                const float ox = __shfl_xor_sync(0xffffffffu, v[s].x, m), oy = __shfl_xor_sync(0xffffffffu, v[s].y, m);
                const float2 t = cmul_conj(make_float2(ox - v[s].x, oy - v[s].y), w);
                v[s] = second ? t : make_float2(v[s].x + ox, v[s].y + oy);
            }
        }
    }
}

// rows: global -> transform along y -> shared memory, row k at brev(k) for the
// z transform
template <int N>
__device__ __forceinline__ void plane_y_fwd(const float2 *Sp, float2 *P, int nz, int lgz, int nys, const float2 *tw) {
    using T = LineOf<N>;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, e = lane & (T::L - 1);
    for (int k0 = (threadIdx.x >> 5) * T::W; k0 < nz; k0 += nw * T::W) {
        const int k = k0 + lane / T::L;
        float2 v[T::V];
#pragma unroll
        for (int s = 0; s < T::V; ++s) v[s] = k < nz ? Sp[k * N + line_brev<N>(e + 32 * s)] : make_float2(0.0f, 0.0f);
        line_dit_fwd<N>(v, tw, lane);
        if (k < nz) {
            float2 *row = P + bitrev(k, lgz) * nys;
#pragma unroll
            for (int s = 0; s < T::V; ++s) row[e + 32 * s] = v[s];
        }
    }
}

// columns: transform along z, divide, transform back, in registers
template <int N>
__device__ __forceinline__ void plane_z(float2 *P, int ny, int nys, const float2 *tw, const float *kxy, const float *kz2,
                                        float lhs0, float lhs1, float inv_ntot) {
    using T = LineOf<N>;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, e = lane & (T::L - 1);
    for (int j0 = (threadIdx.x >> 5) * T::W; j0 < ny; j0 += nw * T::W) {
        const int j = j0 + lane / T::L;
        float2 v[T::V];
#pragma unroll
        for (int s = 0; s < T::V; ++s) v[s] = j < ny ? P[(e + 32 * s) * nys + j] : make_float2(0.0f, 0.0f);
        line_dit_fwd<N>(v, tw, lane);
        const float ky = j < ny ? kxy[j] : 0.0f;
#pragma unroll
        for (int s = 0; s < T::V; ++s) {
            const float lhs = __fmaf_rn(lhs1, __fadd_rn(ky, kz2[e + 32 * s]), lhs0);
            const float sc = fabsf(lhs) < 1.0e-16f ? 0.0f : inv_ntot / lhs;
            v[s] = make_float2(v[s].x * sc, v[s].y * sc);
        }
        line_dif_inv<N>(v, tw, lane);
        if (j < ny)
#pragma unroll
            for (int s = 0; s < T::V; ++s) P[(e + 32 * s) * nys + j] = v[s];
    }
}

// rows: shared memory -> inverse transform along y -> global (row r holds
// plane brev(r))
template <int N>
__device__ __forceinline__ void plane_y_inv(float2 *Sp, const float2 *P, int nz, int lgz, int nys, const float2 *tw) {
    using T = LineOf<N>;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, e = lane & (T::L - 1);
    for (int r0 = (threadIdx.x >> 5) * T::W; r0 < nz; r0 += nw * T::W) {
        const int r = r0 + lane / T::L;
        float2 v[T::V];
#pragma unroll
        for (int s = 0; s < T::V; ++s) v[s] = r < nz ? P[r * nys + e + 32 * s] : make_float2(0.0f, 0.0f);
        line_dif_inv<N>(v, tw, lane);
        if (r < nz) {
            float2 *row = Sp + bitrev(r, lgz) * N;
#pragma unroll
            for (int s = 0; s < T::V; ++s) row[line_brev<N>(e + 32 * s)] = v[s];
        }
    }
}

// shared memory: the plane (rows of ny + 1, an odd stride), both twiddle tables
// and both wavenumber tables
inline size_t plane_periodic_smem(int ny, int nz) { return (size_t)8 * (ny + 1) * nz + (size_t)12 * (ny + nz); }

// Warp transforms of whole lines: the plane passes shared memory twice (after
// the y transform and after the z round trip) where radix-2 stages in shared
// memory passed it once per stage; the butterflies and their order are the
// same, and so are the bits.  One CTA per kx (nx/2 + 1 of 152 SMs).  Step of a
// 64^3 box: 199 us with the stages in shared memory (33.8 us a launch), 126 now.
__global__ void __launch_bounds__(1024, 1) k_plane_periodic(float2 *S, int ny, int nz, int lgy, int lgz, PlaneSpec ps) {
    extern __shared__ unsigned char smem_raw[];
    const int nys = ny + 1;
    float2 *P = reinterpret_cast<float2 *>(smem_raw);    // [k][j]
    float2 *twy = P + (size_t)nys * nz, *twz = twy + ny;
    float *kxy = reinterpret_cast<float *>(twz + nz), *kz2 = kxy + ny;
    const int kx = blockIdx.x;
    float2 *Sp = S + (size_t)kx * nz * ny;
    const float k2x = ps.kx2[kx];
    for (int q = threadIdx.x; q < ny; q += blockDim.x) {
        twy[q] = ps.twy[q];
        kxy[q] = k2x + ps.ky2[q];
    }
    for (int q = threadIdx.x; q < nz; q += blockDim.x) {
        twz[q] = ps.twz[q];
        kz2[q] = ps.kz2[q];
    }
    __syncthreads();
    switch (lgy) {
    case 2: plane_y_fwd<4>(Sp, P, nz, lgz, nys, twy); break;
    case 3: plane_y_fwd<8>(Sp, P, nz, lgz, nys, twy); break;
    case 4: plane_y_fwd<16>(Sp, P, nz, lgz, nys, twy); break;
    case 5: plane_y_fwd<32>(Sp, P, nz, lgz, nys, twy); break;
    case 6: plane_y_fwd<64>(Sp, P, nz, lgz, nys, twy); break;
    case 7: plane_y_fwd<128>(Sp, P, nz, lgz, nys, twy); break;
    case 8: plane_y_fwd<256>(Sp, P, nz, lgz, nys, twy); break;
    default: plane_y_fwd<512>(Sp, P, nz, lgz, nys, twy); break;
    }
    __syncthreads();
    switch (lgz) {
    case 2: plane_z<4>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 3: plane_z<8>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 4: plane_z<16>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 5: plane_z<32>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 6: plane_z<64>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 7: plane_z<128>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    case 8: plane_z<256>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    default: plane_z<512>(P, ny, nys, twz, kxy, kz2, ps.lhs0, ps.lhs1, ps.inv_ntot); break;
    }
    __syncthreads();
    switch (lgy) {
    case 2: plane_y_inv<4>(Sp, P, nz, lgz, nys, twy); break;
    case 3: plane_y_inv<8>(Sp, P, nz, lgz, nys, twy); break;
    case 4: plane_y_inv<16>(Sp, P, nz, lgz, nys, twy); break;
    case 5: plane_y_inv<32>(Sp, P, nz, lgz, nys, twy); break;
    case 6: plane_y_inv<64>(Sp, P, nz, lgz, nys, twy); break;
    case 7: plane_y_inv<128>(Sp, P, nz, lgz, nys, twy); break;
    case 8: plane_y_inv<256>(Sp, P, nz, lgz, nys, twy); break;
    default: plane_y_inv<512>(Sp, P, nz, lgz, nys, twy); break;
    }
}

// Pivot table of the y systems of one solve type: for each (kx, kz) the
// Thomas factors 1/den_j (0 where the pivot vanishes, the reference's guard),
// computed on the host in FP64.  The back-substitution multipliers are
// P_j = -b_j / den_j with b_j the super-diagonal of row j.
struct WallTables {
    const float *rden;   // [kx][kz][j]
    float bc;            // interior off-diagonal b = c
    float c_last;        // c of the last row (1 U, -1 P); V: rows >= ny are identities
    float b_first;       // b of row 0 (1 U, -1 P, 0 V)
    float nxz_inv;
    int sys;
    WallLayout wl;       // shared-memory strides and Thomas rows per thread (wall_layout)
};

// ---------------------------------------------------------------------------
// x passes of XW_RB rows per block (NX = 32 .. 512).  Two real rows are one
// complex line, held by G threads with E elements each: the spans of G and more
// run in registers on the elements t + G s, the rest after one exchange through
// shared memory on the groups of G consecutive elements (NX = 128 and 512: on half
// of a group, with the last span between lanes).  The block then
// unpacks the half spectra of its rows from (packs them into) the lines while
// it writes (reads) the [kx][row] lines of 16 consecutive rows, the two rows of
// a pair on neighbouring lanes.  Bound by instruction issue and shared memory:
// with a warp per line, lane exchanges in the spans below 32 and a second
// shared tile between the lines and the rows, 256x128x128 took 12.8 us forward and
// 15.0 us inverse, this form 9.0 and 10.7 us.
constexpr int XW_RB = 16;     // rows per block of the x passes (a constant: the tile indexing divides by it)

template <int N> struct XLine {
    static constexpr int E = N >= 256 ? 16 : 8, G = N / E, THREADS = XW_RB / 2 * G;
    static constexpr bool PAIRS = G == 2 * E;      // NX = 128, 512
    static constexpr int LG = N == 32 ? 5 : N == 64 ? 6 : N == 128 ? 7 : N == 256 ? 8 : 9;
    // element e of a line at e + PAD (e / G), lines PITCH apart (odd): strided
    // and consecutive elements, and one element of the lines, in distinct banks
    static constexpr int PAD = PAIRS ? 2 : 1, PITCH = N + PAD * E + 1;
    static constexpr size_t smem = (size_t)(N + XW_RB / 2 * PITCH) * sizeof(float2);
    static __device__ __forceinline__ int ix(int e) { return e + e / G * PAD; }
    static __device__ __forceinline__ int at(int k) { return ix((int)(__brev((unsigned)k) >> (32 - LG))); }   // X[k]
};

// spans below G of a line in shared memory (in place), forward or inverse
template <int N, bool FWD>
__device__ __forceinline__ void x_inner(float2 *z, const float2 *tws, int t) {
    using X = XLine<N>;
    if constexpr (X::PAIRS) {
        float2 *x = z + X::ix(t / 2 * X::G) + (t & 1);
        float2 v[X::E];
        const float sg = t & 1 ? -1.0f : 1.0f;
        auto last = [&] {                 // first: a + b, second: a - b
#pragma unroll
            for (int s = 0; s < X::E; ++s) {
                const float ox = __shfl_xor_sync(0xffffffffu, v[s].x, 1), oy = __shfl_xor_sync(0xffffffffu, v[s].y, 1);
                v[s] = __ffma2_rn(make_float2(sg, sg), v[s], make_float2(ox, oy));
            }
        };
#pragma unroll
        for (int s = 0; s < X::E; ++s) v[s] = x[2 * s];
        if (FWD) { reg_dif<X::E, 2>(v, tws, t & 1); last(); }
        else { last(); reg_dit<X::E, 2>(v, tws, t & 1); }
#pragma unroll
        for (int s = 0; s < X::E; ++s) x[2 * s] = v[s];
    } else {
#pragma unroll
        for (int u = 0; u < X::E / X::G; ++u) {
            float2 *x = z + X::ix((t + X::G * u) * X::G);
            float2 v[X::G];
#pragma unroll
            for (int s = 0; s < X::G; ++s) v[s] = x[s];
            if (FWD) reg_dif<X::G, 1>(v, tws, 0);
            else reg_dit<X::G, 1>(v, tws, 0);
#pragma unroll
            for (int s = 0; s < X::G; ++s) x[s] = v[s];
        }
    }
}

template <int N, typename TS>
__global__ void __launch_bounds__(XLine<N>::THREADS) k_xfwd_w(const TS *__restrict__ src, float2 *__restrict__ S, int ny,
                                                             int nz, int lj, int joff, const float2 *__restrict__ twx) {
    using X = XLine<N>;
    constexpr int E = X::E, G = X::G, NH = N / 2;
    extern __shared__ unsigned char smem_raw[];
    float2 *tws = reinterpret_cast<float2 *>(smem_raw);
    float2 *zb = tws + N;
    const int p = threadIdx.x / G, t = threadIdx.x % G;
    float2 *z = zb + p * X::PITCH;
    const int bpp = (ny + XW_RB - 1) / XW_RB;
    const int k = blockIdx.x / bpp;
    const int r0 = (blockIdx.x % bpp) * XW_RB;
    const int nrows = min(XW_RB, ny - r0);
    const bool has_a = 2 * p < nrows, has_b = 2 * p + 1 < nrows;
    const TS *ra = src + (size_t)N * ((size_t)(r0 + 2 * p) + (size_t)ny * k) + t;
    float2 v[E];
#pragma unroll
    for (int s = 0; s < E; ++s)
        v[s] = make_float2(has_a ? (float)ra[G * s] : 0.0f, has_b ? (float)ra[N + G * s] : 0.0f);
    for (int q = threadIdx.x; q < N; q += X::THREADS) tws[q] = twx[q];
    __syncthreads();
    reg_dif<E, G>(v, tws, t);
#pragma unroll
    for (int s = 0; s < E; ++s) z[X::ix(G * s) + t] = v[s];
    __syncwarp();
    x_inner<N, true>(z, tws, t);
    __syncthreads();
    const int r = threadIdx.x % XW_RB, b = r & 1;
    const float2 *zr = zb + (r >> 1) * X::PITCH;
    float2 *Sr = S + (size_t)k * lj + (r0 + r + 1 + joff);
    const int skx = nz * lj;
    if (r < nrows) {
#pragma unroll 4
        for (int kx = threadIdx.x / XW_RB; kx <= NH; kx += X::THREADS / XW_RB) {
            const float2 zk = zr[X::at(kx)], zm = zr[X::at((N - kx) & (N - 1))];
            // A = (zk + conj zm) / 2, B = (zk - conj zm) / 2i
            const float ax = b ? zk.y : zk.x, bx = b ? zm.y : zm.x, ay = b ? zm.x : zk.y, by = b ? zk.x : zm.y;
            Sr[(size_t)kx * skx] = make_float2((ax + bx) * 0.5f, (ay - by) * 0.5f);
        }
    }
}

template <int N, typename Out>
__global__ void __launch_bounds__(XLine<N>::THREADS) k_xinv_w(const float2 *__restrict__ S, Out out, int nrow, int jlo,
                                                             int nz, int lj, int joff2, int sx, int sy,
                                                             const float2 *__restrict__ twx) {
    using X = XLine<N>;
    constexpr int E = X::E, G = X::G, NH = N / 2, STEP = X::THREADS / XW_RB;
    extern __shared__ unsigned char smem_raw[];
    float2 *tws = reinterpret_cast<float2 *>(smem_raw);
    float2 *zb = tws + N;
    const int bpp = (nrow + XW_RB - 1) / XW_RB;
    const int k = blockIdx.x / bpp;
    const int r0 = (blockIdx.x % bpp) * XW_RB;
    const int nrows = min(XW_RB, nrow - r0);
    for (int q = threadIdx.x; q < N; q += X::THREADS) tws[q] = twx[q];
    {
        // Z = A + i B over the full line from the two half spectra: the lane of
        // row a writes Z[kx], that of row b Z[N - kx]
        const int r = threadIdx.x % XW_RB, b = r & 1;
        float2 *zr = zb + (r >> 1) * X::PITCH;
        const float2 *Sr = S + (size_t)k * lj + (jlo + r0 + r + joff2);
        const int skx = nz * lj;
        auto put = [&](int kx, float2 v, bool keep) {
            const float ox = __shfl_xor_sync(0xffffffffu, v.x, 1), oy = __shfl_xor_sync(0xffffffffu, v.y, 1);
            const float2 zv = make_float2((b ? v.y : v.x) + (b ? ox : -oy), (b ? v.x : v.y) + (b ? -oy : ox));
            if (keep && !(b && (kx == 0 || kx == NH))) zr[X::at(b ? N - kx : kx)] = zv;
        };
        const bool first = threadIdx.x < XW_RB;      // kx = NH, by the first lanes of the first warp
        const float2 vl = first && r < nrows ? Sr[(size_t)NH * skx] : make_float2(0.f, 0.f);
        const int k0 = threadIdx.x / XW_RB;          // NH = E STEP: all loads of the tile in flight at once
        float2 v[E];
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = r < nrows ? Sr[(size_t)(k0 + u * STEP) * skx] : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < E; ++u) put(k0 + u * STEP, v[u], true);
        if (threadIdx.x < 32) put(NH, vl, first);
    }
    __syncthreads();
    const int p = threadIdx.x / G, t = threadIdx.x % G;
    float2 *z = zb + p * X::PITCH;
    x_inner<N, false>(z, tws, t);
    __syncwarp();
    float2 v[E];
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = z[X::ix(G * s) + t];
    reg_dit<E, G>(v, tws, t);
    const bool has_a = 2 * p < nrows, has_b = 2 * p + 1 < nrows;
    const size_t oa = 1 + (size_t)sx * ((size_t)(jlo + r0 + 2 * p) + (size_t)sy * (k + 1)) + t;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        if (has_a) out.put(oa + G * s, v[s].x);
        if (has_b) out.put(oa + sx + G * s, v[s].y);
    }
}

// Wall plane with the Thomas solves split over T = 1024 / NZ threads per
// (kx, kz) system and, for planes larger than one CTA's shared memory, over a
// thread-block cluster of cl CTAs holding consecutive bands of y rows.  Both
// sweeps are first-order affine recurrences,
//   forward   q_j = alpha_j q_{j-1} + beta_j,  alpha_j = -c_j / den_j,
//                                              beta_j  = d_j / den_j,
//   backward  x_j = P_j x_{j+1} + q_j,          P_j = -b_j / den_j,
// so each thread composes the maps of its chunk of rows, the T threads of a
// system scan the composed maps with shuffles, the CTAs of the cluster
// exchange their composed maps through distributed shared memory, and each
// thread then replays its chunk from its incoming value.  The coefficients
// are those of the sequential Thomas solve (tdma,
// fenep_2d.f90:1145-1177); the 1/den table of the CTA's rows is staged in
// shared memory, its rows in the bit-reversed kz order of the spectrum rows.
// The cluster barriers are hardware barriers; no thread waits on a flag.
//
// The z transforms of the rows are radix-2 passes over registers, V1 and then
// S = NZ / V1 elements of a line per thread, with the lanes of a warp on
// neighbouring rows: global and shared accesses are contiguous, the twiddles
// of a warp are broadcasts, and no lane multiplies for the other half of a
// pair.  The first pass of the forward transform reads the plane from global
// memory and the last of the inverse writes it there (16 loads in flight per
// thread), and the pivot table arrives by asynchronous copies meanwhile.  The
// kernel is bound by instruction issue: a warp per line with lane exchanges
// executed 275 instructions per value of the plane and took 30.0 us at
// 256x128x128 (one CTA per kx), this form takes 20.2 us.
__device__ __forceinline__ void copy_async4(float *smem, const float *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int N> struct ZSplit {
    static constexpr int V1 = N >= 128 ? 16 : 8, S = N / V1;
};

// Exclusive scan of the composed maps (A, B) of the T chunks of each system, in
// order (UP) or from the end, and the map of all chunks to tot[3][NZ].  The
// thread t NZ + row holds the map of chunk t; the threads row T + t scan them
// with shuffles.  sc: WALL_SCAN floats, pitch NZ + NZ / 32 against conflicts.
template <int NZ, bool UP>
__device__ __forceinline__ void wall_scan(float *sc, float *tot, float &A, float2 &B) {
    constexpr int T = 1024 / NZ, W = NZ + NZ / 32, F = T * W;
    const int own = threadIdx.x / NZ * W + threadIdx.x % NZ;
    const int row = threadIdx.x / T, t = threadIdx.x % T, at = t * W + row;
    __syncthreads();   // earlier reads of what lies under sc
    sc[own] = A; sc[F + own] = B.x; sc[2 * F + own] = B.y;
    __syncthreads();
    A = sc[at]; B = make_float2(sc[F + at], sc[2 * F + at]);
#pragma unroll
    for (int o = 1; o < T; o <<= 1) {
        const float Ap = UP ? __shfl_up_sync(0xffffffffu, A, o, T) : __shfl_down_sync(0xffffffffu, A, o, T);
        const float Bx = UP ? __shfl_up_sync(0xffffffffu, B.x, o, T) : __shfl_down_sync(0xffffffffu, B.x, o, T);
        const float By = UP ? __shfl_up_sync(0xffffffffu, B.y, o, T) : __shfl_down_sync(0xffffffffu, B.y, o, T);
        if (UP ? t >= o : t + o < T) { B = make_float2(fmaf(A, Bx, B.x), fmaf(A, By, B.y)); A *= Ap; }
    }
    // the inclusive map of chunk t is the exclusive one of the next
    if (t == (UP ? T - 1 : 0)) { tot[row] = A; tot[NZ + row] = B.x; tot[2 * NZ + row] = B.y; }
    const int nx = (UP ? (t == T - 1 ? 0 : t + 1) : (t == 0 ? T - 1 : t - 1)) * W + row;
    const bool end = t == (UP ? T - 1 : 0);
    __syncwarp();      // the threads of a system lie in one warp
    sc[nx] = end ? 1.0f : A; sc[F + nx] = end ? 0.0f : B.x; sc[2 * F + nx] = end ? 0.0f : B.y;
    __syncthreads();
    A = sc[own]; B = make_float2(sc[F + own], sc[2 * F + own]);
}

template <int V>
__global__ void __launch_bounds__(1024, 1) k_plane_walls_c(float2 *S, int ny, int cl, const float2 *twz,
                                                           WallTables wt) {
    constexpr int NZ = 32 * V;
    constexpr int LG = V == 1 ? 5 : (V == 2 ? 6 : (V == 4 ? 7 : 8));
    namespace cg = cooperative_groups;
    extern __shared__ unsigned char smem_raw[];
    const int lj = ny + 2;
    const int R = wall_rows_per_cta(lj, cl);
    const int rank = cl > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int kx = blockIdx.x / cl;
    const int jlo = rank * R;
    const int nr = max(0, min(R, lj - jlo));   // rows held by this CTA
    const int ps = wt.wl.ps;
    const int rs = wt.wl.rs;
    float2 *P = reinterpret_cast<float2 *>(smem_raw);                 // [k][jl]
    float *Rs = reinterpret_cast<float *>(P + (size_t)ps * NZ);       // [row][jl], row = bitrev(kz)
    float2 *tws = reinterpret_cast<float2 *>(Rs + (size_t)rs * NZ);   // NZ stage-major twiddles
    float *mapF = reinterpret_cast<float *>(tws + NZ);                // [3][NZ]: A, Bx, By
    float *mapB = mapF + 3 * NZ;
    constexpr int V1 = ZSplit<NZ>::V1, S1 = ZSplit<NZ>::S;
    float *sc = wall_scan_in_plane(ps, NZ) ? reinterpret_cast<float *>(P) : mapB + 3 * NZ;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    float2 *Sp = S + (size_t)kx * NZ * lj + jlo;
    const float *Rg = wt.rden + (size_t)kx * NZ * lj + jlo;
    const bool sysv = wt.sys == SYS_V;
    for (int q = threadIdx.x; q < NZ; q += blockDim.x) tws[q] = twz[q];
    for (int k = warp; k < NZ; k += nwarp) {
        float *rrow = Rs + (size_t)(__brev((unsigned)k) >> (32 - LG)) * rs;
        for (int jl = lane; jl < nr; jl += 32) copy_async4(rrow + jl, Rg + k * lj + jl);
    }
    copy_async_commit();
    // ghost rows, and the row of V on the upper wall, carry no right-hand side
    for (int q = threadIdx.x; q < 3 * NZ; q += blockDim.x) {
        const int j = q < NZ ? 0 : (q < 2 * NZ ? ny : ny + 1), jl = j - jlo;
        if (jl >= 0 && jl < nr && (j != ny || sysv)) P[(q & (NZ - 1)) * ps + jl] = make_float2(0.f, 0.f);
    }
    const int f0 = max(0, 1 - jlo), nf = max(0, min(nr, ny + (sysv ? 0 : 1) - jlo) - f0);   // rows to transform
    __syncthreads();   // twiddles
    for (int q = threadIdx.x; q < nf * S1; q += blockDim.x) {
        const int t = q / nf, jl = f0 + q - t * nf;
        float2 v[V1];
#pragma unroll
        for (int s = 0; s < V1; ++s) v[s] = Sp[(t + S1 * s) * lj + jl];
        reg_dif<V1, S1>(v, tws, t);
#pragma unroll
        for (int s = 0; s < V1; ++s) P[(t + S1 * s) * ps + jl] = v[s];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nf * V1; q += blockDim.x) {
        const int u = q / nf, jl = f0 + q - u * nf;
        float2 *x = P + u * S1 * ps + jl;
        float2 v[S1];
#pragma unroll
        for (int s = 0; s < S1; ++s) v[s] = x[s * ps];
        reg_dif<S1, 1>(v, tws, 0);
#pragma unroll
        for (int s = 0; s < S1; ++s) x[s * ps] = v[s];
    }
    copy_async_wait();
    __syncthreads();
    {
        const int row = threadIdx.x % NZ, t = threadIdx.x / NZ;   // one chunk number per warp
        const int L = wt.wl.L;
        const int c0 = min(nr, t * L), n = min(nr, c0 + L) - c0;
        float2 *x = P + row * ps + c0;
        const float *rd = Rs + row * rs + c0;
        // rows of the chunk with the interior's coefficients; behind them the
        // last row (V: also the row on the wall), where d = 0 and b = 0
        const int nin = min(n, (sysv ? ny : ny + 1) - jlo - c0);
        const float nbc = -wt.bc, nlast = sysv ? -0.0f : -wt.c_last;
        const float nb0 = jlo + c0 == 0 ? -wt.b_first : nbc;
        float2 v[WALL_CHUNK];
        // forward: compose the chunk's maps (row 0 has no predecessor: q = 0)
        float A = 1.0f;
        float2 B = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < WALL_CHUNK; ++i) {
            if (i >= n) break;
            v[i] = x[i];
            const float r = rd[i], al = (i < nin ? nbc : nlast) * r, dr = wt.nxz_inv * r;
            B = make_float2(fmaf(al, B.x, v[i].x * dr), fmaf(al, B.y, v[i].y * dr));
            A *= al;
        }
        wall_scan<NZ, true>(sc, mapF, A, B);
        float2 q = make_float2(0.f, 0.f);
        if (cl > 1) {
            cg::this_cluster().sync();
            for (int rr = 0; rr < rank; ++rr) {
                const float *m = cg::this_cluster().map_shared_rank(mapF, rr);
                const float a = m[row];
                q = make_float2(fmaf(a, q.x, m[NZ + row]), fmaf(a, q.y, m[2 * NZ + row]));
            }
        }
        q = make_float2(fmaf(A, q.x, B.x), fmaf(A, q.y, B.y));
#pragma unroll
        for (int i = 0; i < WALL_CHUNK; ++i) {
            if (i >= n) break;
            const float r = rd[i], al = (i < nin ? nbc : nlast) * r, dr = wt.nxz_inv * r;
            q = make_float2(fmaf(al, q.x, v[i].x * dr), fmaf(al, q.y, v[i].y * dr));
            v[i] = q;
        }
        // backward: x_j = P_j x_{j+1} + q_j (b and so P of the rows behind the
        // interior are 0; row 0 has its own b)
        A = 1.0f;
        B = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = WALL_CHUNK - 1; i >= 0; --i) {
            if (i >= n) continue;
            const float pj = (i >= nin ? -0.0f : (i == 0 ? nb0 : nbc)) * rd[i];
            B = make_float2(fmaf(pj, B.x, v[i].x), fmaf(pj, B.y, v[i].y));
            A *= pj;
        }
        wall_scan<NZ, false>(sc, mapB, A, B);
        q = make_float2(0.f, 0.f);
        if (cl > 1) {
            cg::this_cluster().sync();
            for (int rr = cl - 1; rr > rank; --rr) {
                const float *m = cg::this_cluster().map_shared_rank(mapB, rr);
                const float a = m[row];
                q = make_float2(fmaf(a, q.x, m[NZ + row]), fmaf(a, q.y, m[2 * NZ + row]));
            }
        }
        q = make_float2(fmaf(A, q.x, B.x), fmaf(A, q.y, B.y));
        __syncthreads();   // every thread has read its map: the scan buffer lies in the plane
#pragma unroll
        for (int i = WALL_CHUNK - 1; i >= 0; --i) {
            if (i >= n) continue;
            const float pj = (i >= nin ? -0.0f : (i == 0 ? nb0 : nbc)) * rd[i];
            q = make_float2(fmaf(pj, q.x, v[i].x), fmaf(pj, q.y, v[i].y));
            x[i] = q;
        }
    }
    // the other CTAs' reads of this CTA's maps are complete past this barrier
    if (cl > 1) cg::this_cluster().sync();
    else __syncthreads();
    for (int q = threadIdx.x; q < nr * V1; q += blockDim.x) {
        const int u = q / nr, jl = q - u * nr;
        float2 *x = P + u * S1 * ps + jl;
        float2 v[S1];
#pragma unroll
        for (int s = 0; s < S1; ++s) v[s] = x[s * ps];
        reg_dit<S1, 1>(v, tws, 0);
#pragma unroll
        for (int s = 0; s < S1; ++s) x[s * ps] = v[s];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nr * S1; q += blockDim.x) {
        const int t = q / nr, jl = q - t * nr;
        float2 v[V1];
#pragma unroll
        for (int s = 0; s < V1; ++s) v[s] = P[(t + S1 * s) * ps + jl];
        reg_dit<V1, S1>(v, tws, t);
#pragma unroll
        for (int s = 0; s < V1; ++s) Sp[(t + S1 * s) * lj + jl] = v[s];
    }
}

}  // namespace f8
