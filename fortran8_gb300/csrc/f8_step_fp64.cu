// f8_step_fp64.cu — FP64 kernels of the SMAC + FENE-P + IBM step.
//
// Compiled with --fmad=false: every a*b+c stays two rounded operations, in the
// order the reference writes them, so results can be compared with the CPU
// oracle at the 1e-10 level (and are bit-identical wherever no
// transcendental function is involved).  The cited lines are in
// machapin/fortran8.
#include <algorithm>
#include <cstdio>
#include "f8_common.cuh"
#include "f8_fft.cuh"
#include "f8_kernels.h"
#include "f8_recip.cuh"
#include "f8_sor.cuh"

namespace f8 {

namespace {

constexpr double PI_D = 3.141592653589793238462643383279502884;

// ---------------------------------------------------------------------------
// Halo fill (PBM / C_PBM, fenep.f90:147-166; walls fenep_2d.f90:1098-1143).
// Each halo cell takes its value from an interior cell after wrapping the
// periodic directions, which is what the reference's plane-by-plane copies
// produce.

__device__ inline double halo_value(const Geo &g, const double *A, int kind, int i, int j, int k) {
    const int ii = wrapx(g, i), kk = wrapz(g, k);
    if (j >= 1 && j <= g.ny) {
        if (g.walls && kind == BC_V && j == g.ny) return 0.0;
        return A[hix(g, ii, j, kk)];
    }
    if (!g.walls) return A[hix(g, ii, wrapy(g, j), kk)];
    const bool lo = j == 0;
    switch (kind) {
    case BC_U: return lo ? -A[hix(g, ii, 1, kk)] : 2 * g.uwall - A[hix(g, ii, g.ny, kk)];
    case BC_W: return lo ? -A[hix(g, ii, 1, kk)] : -A[hix(g, ii, g.ny, kk)];
    case BC_V: return 0.0;
    case BC_P: return lo ? A[hix(g, ii, 1, kk)] : A[hix(g, ii, g.ny, kk)];
    default:   return lo ? 2 * A[hix(g, ii, 1, kk)] - A[hix(g, ii, 2, kk)]
                         : 2 * A[hix(g, ii, g.ny, kk)] - A[hix(g, ii, g.ny - 1, kk)];
    }
}

// Boundary values of up to four fields in one launch, and V = 0 on the upper
// wall face (V(:,NB) = 0, fenep_2d.f90:1114)
struct BcSetD {
    double *A[4];
    int kind[4];
    int n;
};

__global__ void k_bc_set64(BcSetD b, Geo g) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (halo_cell(g, t, i, j, k)) {
        const int h = hix(g, i, j, k);
        // every field's source value before the first store
        double v[4];
#pragma unroll
        for (int f = 0; f < 4; ++f)
            if (f < b.n) v[f] = halo_value(g, b.A[f], b.kind[f], i, j, k);
#pragma unroll
        for (int f = 0; f < 4; ++f)
            if (f < b.n) b.A[f][h] = v[f];
        return;
    }
    if (g.walls) {
        t -= halo_count(g);
        if (t >= 0 && t < (long)g.nx * g.nz) {
            i = 1 + (int)(t % g.nx); k = 1 + (int)(t / g.nx);
#pragma unroll
            for (int f = 0; f < 4; ++f)
                if (f < b.n && b.kind[f] == BC_V) b.A[f][hix(g, i, g.ny, k)] = 0.0;
        }
    }
}

// Peterlin factor (fenep.f90:510-515, fenep_2d.f90:275-280).
__device__ inline double peterlin(const double *x, int ncomp, double lp2) {
    return ncomp == 6 ? (lp2 - 3) / (lp2 - x[0] - x[3] - x[5]) : (lp2 - 2) / (lp2 - x[0] - x[2]);
}

// Halo fill of the SoA conformation tensor plus the Peterlin factor of every
// halo cell (the interior f is written by the polymer update).
__global__ void k_bc_c_pet(double *C, double *fpet, Geo g, int ncomp, int cs, double lp2) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!halo_cell(g, t, i, j, k)) return;
    const int h = hix(g, i, j, k);
    double x[6];
    for (int m = 0; m < ncomp; ++m) {
        x[m] = halo_value(g, C + (size_t)m * cs, BC_C, i, j, k);
        C[(size_t)m * cs + h] = x[m];
    }
    fpet[h] = peterlin(x, ncomp, lp2);
}

// After the polymer update of a wall channel: the x and z halo cells of every
// row (ghost rows included) as periodic copies and their Peterlin factor; the
// ghost rows keep their updated values (C_PBM after Lyapunov,
// fenep_2d.f90:348; the wall extrapolation comes at the end of the step).
__global__ void k_bc_c_pet_xz(double *C, double *fpet, Geo g, int ncomp, int cs, double lp2) {
    long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (!halo_cell(g, t, i, j, k)) return;
    if ((j == 0 || j == g.sy - 1) && i >= 1 && i <= g.nx && k >= 1 && k <= g.nz) return;   // updated ghost cell
    const int src = hix(g, wrapx(g, i), j, wrapz(g, k));
    const int h = hix(g, i, j, k);
    double x[6];
    for (int m = 0; m < ncomp; ++m) {
        x[m] = C[(size_t)m * cs + src];
        C[(size_t)m * cs + h] = x[m];
    }
    fpet[h] = peterlin(x, ncomp, lp2);
}

// f on every cell (after a load, or when the polymer stage is skipped)
__global__ void k_pet_all(const double *C, double *fpet, int ncomp, int cs, double lp2) {
    int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= cs) return;
    double x[6];
    for (int m = 0; m < ncomp; ++m) x[m] = C[(size_t)m * cs + h];
    fpet[h] = peterlin(x, ncomp, lp2);
}

// ---------------------------------------------------------------------------
// Polymer, 3D.  Eigen test (Vieta, fenep.f90:425-444) and candidate selection
// (CpxCnx, fenep.f90:169-242).

__device__ inline double vieta(const double *a) {
    double a2 = -(a[0] + a[3] + a[5]);
    double a1 = a[0] * a[3] + a[3] * a[5] + a[5] * a[0] - a[4] * a[4] - a[2] * a[2] - a[1] * a[1];
    double a0 = -(a[0] * a[3] * a[5] + a[1] * a[4] * a[2] + a[1] * a[4] * a[2] - a[0] * a[4] * a[4]
                  - a[1] * a[1] * a[5] - a[2] * a[3] * a[2]);
    double p = a1 - (a2 * a2) / 3.0;
    double q = a0 - a1 * a2 / 3.0 + 2.0 * (a2 * a2 * a2) / 27.0;
    double qh = q / 2.0, p3 = p / 3.0;
    double t = qh * qh + p3 * p3 * p3;
    if (t >= 0.0) return -100.0;
    const double two_pi_3 = 2.0 * PI_D / 3.0;
    return 2.0 * sqrt(-p / 3.0) * cos(acos(3.0 * q / (2.0 * p) * sqrt(-3.0 / p)) / 3.0 + two_pi_3) - a2 / 3.0;
}

__device__ inline double nanmin2(double a, double b) {
    if (isnan(a)) return b;
    if (isnan(b)) return a;
    return b < a ? b : a;
}

// maxloc(minlist, 1) over four values, NaN ignored, first maximum wins.
__device__ inline int maxloc4(const double *m) {
    int idx = 0; double best = 0; bool found = false;
    for (int l = 0; l < 4; ++l) {
        if (isnan(m[l])) continue;
        if (!found || m[l] > best) { best = m[l]; idx = l; found = true; }
    }
    return found ? idx + 1 : 1;
}

// candidate faces of fenep.f90:179-184 (idx 1..3), or the cell value (idx 4)
__device__ inline double face_p(int idx, double cm, double c0, double cp) {
    switch (idx) {
    case 1: return c0 * 3 / 2 - cp / 2;
    case 2: return cm / 2 + c0 / 2;
    case 3: return cm / 4 + c0 - cp / 4;
    default: return c0;
    }
}
__device__ inline double face_n(int idx, double cm, double c0, double cp) {
    switch (idx) {
    case 1: return c0 / 2 + cp / 2;
    case 2: return -cm / 2 + c0 * 3 / 2;
    case 3: return -cm / 4 + c0 + cp / 4;
    default: return c0;
    }
}

// The reference's other eigen tests (its compile-time eigen_method,
// fenep.f90:187-212).  Cardano (fenep.f90:384-423): the three roots from the
// complex cube roots of u3 = -q/2 + i sqrt(-t) and its conjugate; with
// u3 = rho e^(i th) the principal cube roots give 2 rho^(1/3) cos(th/3 + 2 pi
// k/3) - a2/3, k = 0, 1, -1.  The reference sets -1 when t >= 0 (and then
// reads u3, v3 unset; the evident intent, -1, is kept here).
__device__ inline void cardano(const double *a, double *e) {
    double a2 = -(a[0] + a[3] + a[5]);
    double a1 = a[0] * a[3] + a[3] * a[5] + a[5] * a[0] - a[4] * a[4] - a[2] * a[2] - a[1] * a[1];
    double a0 = -(a[0] * a[3] * a[5] + a[1] * a[4] * a[2] + a[1] * a[4] * a[2] - a[0] * a[4] * a[4]
                  - a[1] * a[1] * a[5] - a[2] * a[3] * a[2]);
    double p = a1 - (a2 * a2) / 3.0;
    double q = a0 - a1 * a2 / 3.0 + 2.0 * (a2 * a2 * a2) / 27.0;
    double qh = q / 2.0, p3 = p / 3.0;
    double t = qh * qh + p3 * p3 * p3;
    if (t >= 0.0) { e[0] = e[1] = e[2] = -1.0; return; }
    const double rho = sqrt(qh * qh - t), th = atan2(sqrt(-t), -qh);
    const double r3 = cbrt(rho), two_pi_3 = 2.0 * PI_D / 3.0;
    e[0] = 2.0 * r3 * cos(th / 3.0) - a2 / 3.0;
    e[1] = 2.0 * r3 * cos(th / 3.0 + two_pi_3) - a2 / 3.0;
    e[2] = 2.0 * r3 * cos(th / 3.0 - two_pi_3) - a2 / 3.0;
}

// Sylvester's criterion (fenep.f90:446-461): 1 for positive leading minors, else -1
__device__ inline double sylvester(const double *a) {
    if (a[0] > 0 && a[3] > 0 && a[5] > 0)
        if (a[0] * a[3] - a[1] * a[1] > 0)
            if (a[0] * a[3] * a[5] + a[1] * a[4] * a[2] + a[1] * a[4] * a[2] - a[0] * a[4] * a[4]
                - a[1] * a[1] * a[5] - a[2] * a[3] * a[2] > 0)
                return 1.0;
    return -1.0;
}

// The smallest eigenvalue of the symmetric matrix, repeated roots included
// (the reference's dsyev, fenep.f90:197-212): the trigonometric form of the
// deviator B = A - m I, p2 = |B|^2/6, r = det(B)/2 / p2^(3/2) clamped to
// [-1, 1] (Smith, Comm. ACM 4 (1961) 168).
__device__ inline double symmetric_min(const double *a) {
    const double m = (a[0] + a[3] + a[5]) / 3.0;
    const double b0 = a[0] - m, b3 = a[3] - m, b5 = a[5] - m;
    const double p2 = (b0 * b0 + b3 * b3 + b5 * b5 + 2.0 * (a[1] * a[1] + a[2] * a[2] + a[4] * a[4])) / 6.0;
    if (!(p2 > 0.0)) return p2 == 0.0 ? m : p2;   // p2 NaN: NaN
    const double det = b0 * (b3 * b5 - a[4] * a[4]) - a[1] * (a[1] * b5 - a[4] * a[2]) + a[2] * (a[1] * a[4] - b3 * a[2]);
    double r = det / 2.0 / (p2 * sqrt(p2));
    r = r < -1.0 ? -1.0 : (r > 1.0 ? 1.0 : r);
    return m + 2.0 * sqrt(p2) * cos(acos(r) / 3.0 + 2.0 * PI_D / 3.0);
}

// minval over the values of one candidate's two faces (fenep.f90:186-241)
__device__ inline double face_test(int method, const double *pt, const double *nt) {
    if (method == 1) {
        double e[6];
        cardano(pt, e);
        cardano(nt, e + 3);
        double v = e[0];
        for (int q = 1; q < 6; ++q) v = nanmin2(v, e[q]);
        return v;
    }
    if (method == 2) return nanmin2(sylvester(pt), sylvester(nt));
    if (method == 3) return nanmin2(symmetric_min(pt), symmetric_min(nt));
    return nanmin2(vieta(pt), vieta(nt));
}

__device__ inline int select3(const double *cm, const double *c0, const double *cp, int method) {
    double minlist[4];
    for (int l = 1; l <= 3; ++l) {
        double pt[6], nt[6];
        for (int m = 0; m < 6; ++m) {
            pt[m] = face_p(l, cm[m], c0[m], cp[m]);
            nt[m] = face_n(l, cm[m], c0[m], cp[m]);
        }
        minlist[l - 1] = face_test(method, pt, nt);
    }
    minlist[3] = 0.0;
    return maxloc4(minlist);
}

// C of component array Cm at row jj of column (i, k): zero beyond the ghost
// rows of a wall channel (the wall mode's outside rows)
__device__ inline double crow(const double *Cm, const Geo &g, int i, int jj, int k) {
    return (jj < 0 || jj > g.ny + 1) ? 0.0 : Cm[hix(g, i, jj, k)];
}

// code of cell (i, j, k), interior or ghost row
__device__ inline int code_at(const uint8_t *codes, const uint8_t *codes_g, const Geo &g, int i, int j, int k) {
    return (j >= 1 && j <= g.ny) ? codes[qix(g, i, j, k)] : codes_g[gcix(g, i, j, k)];
}

__global__ void __launch_bounds__(128) k_polymer_codes3(const double *__restrict__ C, uint8_t *__restrict__ codes,
                                                        uint8_t *__restrict__ codes_g, Geo g, int cs, int method) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + prow0(g);
    const int k = blockIdx.z + 1;
    if (i > g.nx || j >= prow0(g) + prows(g)) return;
    double c0[6], cm[6], cp[6];
    const int h = hix(g, i, j, k);
    for (int m = 0; m < 6; ++m) c0[m] = C[(size_t)m * cs + h];
    const int off[3] = {1, g.sx, g.sx * g.sy};
    int code = 0;
    for (int d = 0; d < 3; ++d) {
        for (int m = 0; m < 6; ++m) {
            if (d == 1 && g.walls) {
                cm[m] = crow(C + (size_t)m * cs, g, i, j - 1, k);
                cp[m] = crow(C + (size_t)m * cs, g, i, j + 1, k);
            } else {
                cm[m] = C[(size_t)m * cs + h - off[d]];
                cp[m] = C[(size_t)m * cs + h + off[d]];
            }
        }
        code |= (select3(cm, c0, cp, method) - 1) << (2 * d);
    }
    if (j >= 1 && j <= g.ny) codes[qix(g, i, j, k)] = (uint8_t)code;
    else codes_g[gcix(g, i, j, k)] = (uint8_t)code;
}

// The queue of k_codes3_filter: the FP64 evaluation of the (cell, direction)
// pairs whose choice rounding might change.  Two lanes per entry, one for each
// face of a candidate, so that a short queue's FP64 chain (three Vieta
// evaluations, ~170 FP64 slots each) is half as long.
__global__ void __launch_bounds__(128) k_codes3_exact(const double *__restrict__ C, uint8_t *codes, uint8_t *codes_g,
                                                      Geo g, int cs, const unsigned *__restrict__ q0,
                                                      const unsigned *__restrict__ q1, const unsigned *__restrict__ q2,
                                                      const int *__restrict__ count) {
    const int n0 = count[0], n1 = count[1], n = n0 + n1 + count[2];
    const int face = threadIdx.x & 1;
    // whole warps stay in the loop together for the shuffles
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 1; (w & ~15) < n; w += (gridDim.x * blockDim.x) >> 1) {
        const bool active = w < n;
        int d = 0, code = 0;
        unsigned e = 0;
        double v[3] = {0.0, 0.0, 0.0};
        int i = 1, j = 1, k = 1;
        if (active) {
            d = w < n0 ? 0 : (w < n0 + n1 ? 1 : 2);
            e = d == 0 ? q0[w] : (d == 1 ? q1[w - n0] : q2[w - n0 - n1]);
            i = (int)(e % g.nx) + 1;
            const int r = (int)(e / g.nx);
            j = r % prows(g) + prow0(g);
            k = r / prows(g) + 1;
            const int h = hix(g, i, j, k), od = d == 0 ? 1 : (d == 1 ? g.sx : g.sx * g.sy);
            const bool lo = !(d == 1 && j == 0), hi = !(d == 1 && j == g.ny + 1);   // zero beyond the ghost rows
            double c0[6], cm[6], cp[6];
            for (int m = 0; m < 6; ++m) {
                const double *Cm = C + (size_t)m * cs + h;
                c0[m] = Cm[0];
                cm[m] = lo ? Cm[-od] : 0.0;
                cp[m] = hi ? Cm[od] : 0.0;
            }
#pragma unroll 1
            for (int l = 1; l <= 3; ++l) {
                double f[6];
                for (int m = 0; m < 6; ++m)
                    f[m] = face ? face_n(l, cm[m], c0[m], cp[m]) : face_p(l, cm[m], c0[m], cp[m]);
                v[l - 1] = vieta(f);
            }
        }
        double minlist[4];
        for (int l = 0; l < 3; ++l) {
            const double o = __shfl_xor_sync(0xffffffffu, v[l], 1);
            minlist[l] = face ? nanmin2(o, v[l]) : nanmin2(v[l], o);
        }
        minlist[3] = 0.0;
        code = (maxloc4(minlist) - 1) << (2 * d);
        if (active && face == 0 && code) {
            uint8_t *dst = (j >= 1 && j <= g.ny) ? codes + qix(g, i, j, k) : codes_g + gcix(g, i, j, k);
            const size_t a = reinterpret_cast<size_t>(dst);
            atomicOr(reinterpret_cast<unsigned *>(a & ~(size_t)3), (unsigned)code << (8 * (a & 3)));
        }
    }
}

// ---------------------------------------------------------------------------
// Divisors of the polymer update: the reference's expressions with their
// divisions by constants.
struct PolyConst {
    Recip d2[3], d1[3], d4[3];   // 2 dX, dX, 4 dX, ... of the three directions
    Recip wi, dc2;               // Wi, 2 dc
    double dtwi;                 // dt / Wi
    double eps2_lo, eps2_hi;     // bounds of the step test (below)
};

PolyConst poly_const(const Geo &g, const Phys &ph) {
    PolyConst c;
    const double d[3] = {g.dx, g.dy, g.dz};
    for (int q = 0; q < 3; ++q) {
        c.d1[q] = recip(d[q]);
        c.d2[q] = recip(2 * d[q]);
        c.d4[q] = recip(4 * d[q]);
    }
    c.wi = recip(ph.wi);
    c.dc2 = recip(2.0 * ph.newton_dc);
    c.dtwi = ph.dt / ph.wi;
    const bool squared = ph.newton_eps > 1.0e-140 && ph.newton_eps < 1.0e140;
    c.eps2_lo = squared ? ph.newton_eps * ph.newton_eps * (1.0 - 1.0e-12) : 0.0;
    c.eps2_hi = squared ? ph.newton_eps * ph.newton_eps * (1.0 + 1.0e-12) : INFINITY;
    return c;
}

// The same for the stencils of the momentum, projection and IBM kernels
struct GridRecip {
    Recip d1[3], d4[3], dd[3];   // dX, 4 dX, dX^2, ...
    Recip dt;
};

GridRecip grid_recip(const Geo &g) {
    GridRecip c;
    const double d[3] = {g.dx, g.dy, g.dz};
    for (int q = 0; q < 3; ++q) {
        c.d1[q] = recip(d[q]);
        c.d4[q] = recip(4 * d[q]);
        c.dd[q] = recip(d[q] * d[q]);
    }
    c.dt = recip(g.dt);
    return c;
}

// The Newton step test sqrt(sr / sx) < eps (fenep.f90:575).  Squared, away from
// the boundary by more than the rounding of either form; the reference's
// expression within it, for NaN, and for a tolerance that is not positive (all
// itrmax iterations run then) or whose square is out of range.
__device__ __forceinline__ bool newton_small(double sr, double sx, double eps, const PolyConst &c) {
    if (sr < sx * c.eps2_lo) return true;
    if (sr > sx * c.eps2_hi) return false;
    return sqrt(sr / sx) < eps;
}

// A candidate face of fenep.f90:179-184 as w * t, with w a power of two and t
// two rounded operations that give the reference's value scaled by 1/w exactly
// (a scaling by a power of two commutes with rounding): t = RN(RN(a c0 + e) + f).
//   plus face:  1: 3 c0/2 - cp/2 = (RN(3 c0) - cp)/2;  2: cm/2 + c0/2 = (c0 + cm)/2;
//               3: cm/4 + c0 - cp/4 = (RN(4 c0 + cm) - cp)/4;  4: c0
//   minus face: 1: (c0 + cp)/2;  2: (RN(3 c0) - cm)/2;  3: (RN(4 c0 - cm) + cp)/4;  4: c0
// The candidate differs from lane to lane; a switch over the reference's
// expressions costs every lane all of them (11 FP64 slots), this form two.
struct FaceSel {
    double a;        // factor of c0
    double w;        // scale
    int idx;
};
__device__ __forceinline__ FaceSel face_sel(int idx, bool minus) {
    FaceSel s;
    s.a = idx == 3 ? 4.0 : (idx == (minus ? 2 : 1) ? 3.0 : 1.0);
    s.w = idx == 3 ? 0.25 : (idx == 4 ? 1.0 : 0.5);
    s.idx = idx;
    return s;
}
__device__ __forceinline__ double face_pt(const FaceSel &s, double cm, double c0, double cp) {
    const double e = s.idx == 2 || s.idx == 3 ? cm : 0.0, f = s.idx == 1 || s.idx == 3 ? cp : 0.0;
    return __dsub_rn(__fma_rn(c0, s.a, e), f);
}
__device__ __forceinline__ double face_nt(const FaceSel &s, double cm, double c0, double cp) {
    const double e = s.idx == 1 ? cp : (s.idx == 3 ? -cm : 0.0), f = s.idx == 2 ? -cm : (s.idx == 3 ? cp : 0.0);
    return __dadd_rn(__fma_rn(c0, s.a, e), f);
}

// Lyapunov_func (fenep.f90:588-605) and its central-difference Jacobian
// (fenep.f90:540-572): the sums in the reference's order, every product and
// partial sum that a perturbed column leaves unchanged taken from the base point
// (the same operations on the same operands give the same double).
//  * the off-diagonal columns (x1, x2, x4) do not change f(X): the diagonal of A
//    is the base one, one row does not hold the variable (its entry is 0), and
//    the sums before the variable's first term are the base ones;
//  * the diagonal columns (x0, x3, x5) change f(X), so each row from its first
//    diagonal term on.
// About 1,000 FP64 slots an iteration where 13 full evaluations, the divisions
// and the elimination took 1,700.
struct Lyap3 {
    double a01, a02, a10, a12, a20, a21, a00, a11, a22;
};

struct LyapSums {
    double d00, d10, d20, d11, d21, d22;   // (A00+A00), (A11+A00), (A22+A00), ...
};

__device__ __forceinline__ LyapSums lyap_sums(const Lyap3 &A, double x0, double x3, double x5, double lp2, double dt,
                                              const PolyConst &pc) {
    const double fx = (lp2 - 3) / (lp2 - x0 - x3 - x5);
    const double dd = (1.0 + div_by(fx * dt, pc.wi)) * 0.5;
    const double a0 = A.a00 + dd, a1 = A.a11 + dd, a2 = A.a22 + dd;
    return LyapSums{a0 + a0, a1 + a0, a2 + a0, a1 + a1, a2 + a1, a2 + a2};
}

// the products that do not hold a diagonal element of A
struct LyapProd {
    double p01x1, p02x2, p10x0, p12x2, p01x3, p02x4, p20x0, p21x1, p01x4, p02x5, p10x1, p12x4, p10x2, p20x1, p21x3,
        p12x5, p20x2, p21x4;
};

// residuals of all rows with the diagonal sums D and the given diagonal
// variables (x0, x3, x5 may be perturbed; p10x0, p20x0, p01x3, p21x3, p02x5 and
// p12x5 are their products)
__device__ __forceinline__ void lyap_rows(const LyapSums &D, const LyapProd &P, const double (&x)[6], double x0,
                                          double x3, double x5, double p10x0, double p20x0, double p01x3, double p21x3,
                                          double p02x5, double p12x5, const double (&b)[6], double r3, double r5,
                                          double (&l)[6]) {
    l[0] = D.d00 * x0 + P.p01x1 + P.p02x2 + P.p01x1 + P.p02x2 - b[0];
    l[1] = p10x0 + D.d10 * x[1] + P.p12x2 + p01x3 + P.p02x4 - b[1];
    l[2] = p20x0 + P.p21x1 + D.d20 * x[2] + P.p01x4 + p02x5 - b[2];
    l[3] = r3 + D.d11 * x3 + P.p12x4 + P.p12x4 - b[3];
    l[4] = P.p10x2 + P.p20x1 + p21x3 + D.d21 * x[4] + p12x5 - b[4];
    l[5] = r5 + D.d22 * x5 - b[5];
}

// the residual at x in Ah[.][6] and the Jacobian in Ah[.][0..5]
__device__ __forceinline__ void lyap_system(const Lyap3 &A, const double (&b)[6], const double (&x)[6], double lp2,
                                            double dt, double dc, const PolyConst &pc, double (&Ah)[6][7]) {
    LyapProd P;
    P.p01x1 = A.a01 * x[1]; P.p02x2 = A.a02 * x[2]; P.p10x0 = A.a10 * x[0]; P.p12x2 = A.a12 * x[2];
    P.p01x3 = A.a01 * x[3]; P.p02x4 = A.a02 * x[4]; P.p20x0 = A.a20 * x[0]; P.p21x1 = A.a21 * x[1];
    P.p01x4 = A.a01 * x[4]; P.p02x5 = A.a02 * x[5]; P.p10x1 = A.a10 * x[1]; P.p12x4 = A.a12 * x[4];
    P.p10x2 = A.a10 * x[2]; P.p20x1 = A.a20 * x[1]; P.p21x3 = A.a21 * x[3]; P.p12x5 = A.a12 * x[5];
    P.p20x2 = A.a20 * x[2]; P.p21x4 = A.a21 * x[4];
    const LyapSums D = lyap_sums(A, x[0], x[3], x[5], lp2, dt, pc);
    const double r3 = P.p10x1 + P.p10x1, r5 = P.p20x2 + P.p21x4 + P.p20x2 + P.p21x4;
    {
        double l[6];
        lyap_rows(D, P, x, x[0], x[3], x[5], P.p10x0, P.p20x0, P.p01x3, P.p21x3, P.p02x5, P.p12x5, b, r3, r5, l);
#pragma unroll
        for (int r = 0; r < 6; ++r) Ah[r][6] = l[r];
    }
    // columns 0, 3, 5
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int col = c == 0 ? 0 : (c == 1 ? 3 : 5);
        double l1[6], l2[6];
#pragma unroll
        for (int sg = 0; sg < 2; ++sg) {
            const double xv = sg == 0 ? x[col] + dc : x[col] - dc;
            const double x0 = col == 0 ? xv : x[0], x3 = col == 3 ? xv : x[3], x5 = col == 5 ? xv : x[5];
            const LyapSums Dp = lyap_sums(A, x0, x3, x5, lp2, dt, pc);
            lyap_rows(Dp, P, x, x0, x3, x5, col == 0 ? A.a10 * xv : P.p10x0, col == 0 ? A.a20 * xv : P.p20x0,
                      col == 3 ? A.a01 * xv : P.p01x3, col == 3 ? A.a21 * xv : P.p21x3, col == 5 ? A.a02 * xv : P.p02x5,
                      col == 5 ? A.a12 * xv : P.p12x5, b, r3, r5, sg == 0 ? l1 : l2);
        }
#pragma unroll
        for (int r = 0; r < 6; ++r) Ah[r][col] = div_by(l1[r] - l2[r], pc.dc2);
    }
    // columns 1, 2, 4: rows in the reference's order from the variable's first term
    const double q0x0 = D.d00 * x[0], q1x1 = D.d10 * x[1], q2x2 = D.d20 * x[2], q3x3 = D.d11 * x[3],
                 q4x4 = D.d21 * x[4], q5x5 = D.d22 * x[5];
    double v1[5], v2[5];
#pragma unroll
    for (int sg = 0; sg < 2; ++sg) {
        const double y = sg == 0 ? x[1] + dc : x[1] - dc;
        double *v = sg == 0 ? v1 : v2;
        const double t0 = A.a01 * y, t3 = A.a10 * y;
        v[0] = q0x0 + t0 + P.p02x2 + t0 + P.p02x2 - b[0];
        v[1] = P.p10x0 + D.d10 * y + P.p12x2 + P.p01x3 + P.p02x4 - b[1];
        v[2] = P.p20x0 + A.a21 * y + q2x2 + P.p01x4 + P.p02x5 - b[2];
        v[3] = t3 + t3 + q3x3 + P.p12x4 + P.p12x4 - b[3];
        v[4] = P.p10x2 + A.a20 * y + P.p21x3 + q4x4 + P.p12x5 - b[4];
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) Ah[r][1] = div_by(v1[r] - v2[r], pc.dc2);
    Ah[5][1] = 0.0;
    const double s1 = P.p10x0 + q1x1, s2 = P.p20x0 + P.p21x1, s0 = q0x0 + P.p01x1;
#pragma unroll
    for (int sg = 0; sg < 2; ++sg) {
        const double y = sg == 0 ? x[2] + dc : x[2] - dc;
        double *v = sg == 0 ? v1 : v2;
        const double t0 = A.a02 * y, t5 = A.a20 * y;
        v[0] = s0 + t0 + P.p01x1 + t0 - b[0];
        v[1] = s1 + A.a12 * y + P.p01x3 + P.p02x4 - b[1];
        v[2] = s2 + D.d20 * y + P.p01x4 + P.p02x5 - b[2];
        v[3] = A.a10 * y + P.p20x1 + P.p21x3 + q4x4 + P.p12x5 - b[4];
        v[4] = t5 + P.p21x4 + t5 + P.p21x4 + q5x5 - b[5];
    }
    Ah[0][2] = div_by(v1[0] - v2[0], pc.dc2);
    Ah[1][2] = div_by(v1[1] - v2[1], pc.dc2);
    Ah[2][2] = div_by(v1[2] - v2[2], pc.dc2);
    Ah[3][2] = 0.0;
    Ah[4][2] = div_by(v1[3] - v2[3], pc.dc2);
    Ah[5][2] = div_by(v1[4] - v2[4], pc.dc2);
    const double e1 = s1 + P.p12x2 + P.p01x3, e2 = s2 + q2x2, e3 = r3 + q3x3, e4 = P.p10x2 + P.p20x1 + P.p21x3;
#pragma unroll
    for (int sg = 0; sg < 2; ++sg) {
        const double y = sg == 0 ? x[4] + dc : x[4] - dc;
        double *v = sg == 0 ? v1 : v2;
        const double t3 = A.a12 * y, t5 = A.a21 * y;
        v[0] = e1 + A.a02 * y - b[1];
        v[1] = e2 + A.a01 * y + P.p02x5 - b[2];
        v[2] = e3 + t3 + t3 - b[3];
        v[3] = e4 + D.d21 * y + P.p12x5 - b[4];
        v[4] = P.p20x2 + t5 + P.p20x2 + t5 + q5x5 - b[5];
    }
    Ah[0][4] = 0.0;
#pragma unroll
    for (int r = 0; r < 5; ++r) Ah[r + 1][4] = div_by(v1[r] - v2[r], pc.dc2);
}

// magnitude order of two doubles from their high words (sign dropped): true
// only when |a| > |b| whatever the low words are
__device__ __forceinline__ bool surely_larger(double a, double b) {
    return (__double2hiint(a) & 0x7fffffff) > (__double2hiint(b) & 0x7fffffff);
}

// Gauss-Jordan with partial pivoting (fenep.f90:608-643)
template <int N>
__device__ inline void gauss(double (&Ah)[N][N + 1], double *x) {
    for (int k = 0; k < N; ++k) {
        int maxidx = k; double maxabs = fabs(Ah[k][k]);
        for (int r = k + 1; r < N; ++r) {
            double a = fabs(Ah[r][k]);
            if (a > maxabs) { maxabs = a; maxidx = r; }
        }
        if (maxabs == 0.0) {
            for (int r = 0; r < N; ++r) Ah[r][N] = 0.0;
            break;
        }
        if (k != maxidx)
            for (int q = k; q <= N; ++q) { double tmp = Ah[k][q]; Ah[k][q] = Ah[maxidx][q]; Ah[maxidx][q] = tmp; }
        const double piv = Ah[k][k];
        for (int q = k + 1; q <= N; ++q) Ah[k][q] = Ah[k][q] / piv;
        Ah[k][k] = 1.0;
        for (int r = 0; r < N; ++r) {
            if (r == k) continue;
            double f = Ah[r][k];
            for (int q = k + 1; q <= N; ++q) Ah[r][q] = Ah[r][q] - f * Ah[k][q];
            Ah[r][k] = 0.0;
        }
    }
    for (int r = 0; r < N; ++r) x[r] = Ah[r][N];
}

// The same elimination where every pivot is the diagonal element, as nearly
// always (the Lyapunov system is dominated by it): in registers, the pivot
// search as integer comparisons of the high words, the pivot row divided through
// a reciprocal whose second part only needs a few bits.  Returns false, with x
// unusable, when some pivot might be another row's or a value is not finite (an
// infinite or NaN quotient may differ from the division's).
template <int N>
__device__ __forceinline__ bool gauss_diagonal(double (&Ah)[N][N + 1], double *x) {
    bool plain = true;
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
        for (int r = k + 1; r < N; ++r) plain = plain && surely_larger(Ah[k][k], Ah[r][k]);
        const double h = 1.0 / Ah[k][k];
        const Recip piv{h, __dmul_rn(__fma_rn(-Ah[k][k], h, 1.0), h)};
#pragma unroll
        for (int q = k + 1; q <= N; ++q) Ah[k][q] = div_by(Ah[k][q], piv);
#pragma unroll
        for (int r = 0; r < N; ++r)
            if (r != k) {
                const double f = Ah[r][k];
#pragma unroll
                for (int q = k + 1; q <= N; ++q) Ah[r][q] = Ah[r][q] - f * Ah[k][q];
            }
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
        x[r] = Ah[r][N];
        plain = plain && (__double2hiint(x[r]) & 0x7ff00000) != 0x7ff00000;
    }
    return plain && surely_larger(Ah[N - 1][N - 1], 0.0);
}

// The Newton step with the pivoting elimination, out of line
__device__ __noinline__ void lyap_step_pivoting(const Lyap3 &A, const double (&b)[6], const double (&x)[6], double lp2,
                                                double dt, double dc, const PolyConst &pc, double (&r)[6]) {
    double Ah[6][7];
    lyap_system(A, b, x, lp2, dt, dc, pc, Ah);
    gauss<6>(Ah, r);
}

// Cstar (fenep.f90:464-507) + Lyapunov Newton (fenep.f90:518-585) for one
// cell.  The face states Cp/Cn of the three cells along each direction are
// rebuilt from their selection codes, so no face arrays are stored.  Bound by
// the FP64 pipe: one warp instruction holds its sub-partition's pipe for 64
// cycles (as long as its latency), so what counts is the number of FP64 slots,
// not the occupancy; integer selects are free beside it.
template <bool WALLS>
__global__ void __launch_bounds__(128, 2) k_polymer_update3(const double *__restrict__ C, double *__restrict__ Cn,
                                                         double *__restrict__ fpet, const uint8_t *__restrict__ codes,
                                                         const uint8_t *__restrict__ codes_g,
                                                         const double *__restrict__ U, const double *__restrict__ V,
                                                         const double *__restrict__ W, Geo g, Phys ph, PolyConst pc,
                                                         int cs, StepCounters *cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + prow0(g);
    const int k = blockIdx.z + 1;
    const bool active = i <= g.nx && j < prow0(g) + prows(g);
    unsigned long long my_itr = 0, my_unconv = 0;
    if (active) {
        const int h = hix(g, i, j, k);
        const double dt = ph.dt;
        // selection codes of the cell and its neighbours (with walls the rows
        // beyond the ghost rows are outside: their faces are multiplied by
        // exactly zero in Cstar, the code there is the cell value's)
        const int xm = wrapx(g, i - 1), xp = wrapx(g, i + 1), zm = wrapz(g, k - 1), zp = wrapz(g, k + 1);
        int jm = j - 1, jp = j + 1;
        if (!WALLS) { jm = wrapy(g, jm); jp = wrapy(g, jp); }
        const int cself = code_at(codes, codes_g, g, i, j, k);
        const int cym = (WALLS && jm < 0) ? 3 : (code_at(codes, codes_g, g, i, jm, k) >> 2) & 3;
        const int cyp = (WALLS && jp > g.ny + 1) ? 3 : (code_at(codes, codes_g, g, i, jp, k) >> 2) & 3;
        const int ox = 1, oy = g.sx, oz = g.sx * g.sy;
        double b[6], x[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) { x[m] = C[(size_t)m * cs + h]; b[m] = 0.0; }
        // The directions in the reference's order of the sum: per direction the
        // plus face of this cell's minus side, the plus face of the plus
        // neighbour, the minus face of the minus neighbour and this cell's minus
        // face (s3 Cpxm + s1 Cpxp + s4 Cnxm + s2 Cnxp + ...).
        double u00, u11, u22;
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            const double *Vd = d == 0 ? U : (d == 1 ? V : W);
            const int od = d == 0 ? ox : (d == 1 ? oy : oz);
            const int self = ((cself >> (2 * d)) & 3) + 1;
            const int cm_ = d == 0 ? code_at(codes, codes_g, g, xm, j, k) & 3
                                   : (d == 1 ? cym : (code_at(codes, codes_g, g, i, j, zm) >> 4) & 3);
            const int cp_ = d == 0 ? code_at(codes, codes_g, g, xp, j, k) & 3
                                   : (d == 1 ? cyp : (code_at(codes, codes_g, g, i, j, zp) >> 4) & 3);
            const bool ywall = WALLS && d == 1;
            const double v1 = ywall && j == 0 ? 0.0 : Vd[h - od], v2 = Vd[h];
            const Recip r2 = pc.d2[d];
            const double a1 = fabs(v1), a2 = fabs(v2);
            // s1 s2 s3 s4 of fenep.f90:481-492, scaled by the faces' powers of two
            const double t1 = div_by((-v2 + a2) * dt, r2), t2 = 1.0 / 6 + div_by((-v2 - a2) * dt, r2);
            const double t3 = 1.0 / 6 + div_by((v1 - a1) * dt, r2), t4 = div_by((v1 + a1) * dt, r2);
            const FaceSel fps = face_sel(self, false), fns = face_sel(self, true), fpp = face_sel(cp_ + 1, false),
                          fnm = face_sel(cm_ + 1, true);
            const double s3 = t3 * fps.w, s2 = t2 * fns.w, s1 = t1 * fpp.w, s4 = t4 * fnm.w;
            // the neighbours' centres and the cells beyond them (through the
            // periodic image; zero beyond the ghost rows of a wall channel)
            int hm, hp;
            if (d == 0) { hm = hix(g, xm, j, k); hp = hix(g, xp, j, k); }
            else if (d == 1) { hm = ywall ? h - od : hix(g, i, jm, k); hp = ywall ? h + od : hix(g, i, jp, k); }
            else { hm = hix(g, i, j, zm); hp = hix(g, i, j, zp); }
            const bool m1 = !(ywall && j < 1), m2 = !(ywall && j < 2), p1 = !(ywall && j > g.ny), p2 = !(ywall && j > g.ny - 1);
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const double *Cm = C + (size_t)m * cs;
                const double c0 = x[m];
                const double cm = m1 ? Cm[h - od] : 0.0, cp = p1 ? Cm[h + od] : 0.0;
                const double nm = ywall ? cm : Cm[hm], np = ywall ? cp : Cm[hp];      // neighbours' own values
                const double mm = m2 ? Cm[hm - od] : 0.0, pp = p2 ? Cm[hp + od] : 0.0;
                const double mc = ywall ? c0 : Cm[hm + od], pm = ywall ? c0 : Cm[hp - od];
                const double f3 = s3 * face_pt(fps, cm, c0, cp);
                b[m] = d == 0 ? f3 : b[m] + f3;
                b[m] = b[m] + s1 * face_pt(fpp, pm, np, pp);
                b[m] = b[m] + s4 * face_nt(fnm, mm, nm, mc);
                b[m] = b[m] + s2 * face_nt(fns, cm, c0, cp);
            }
            const double du = div_by(-dt * (-v1 + v2), pc.d1[d]);
            if (d == 0) u00 = du;
            else if (d == 1) u11 = du;
            else u22 = du;
        }
        b[0] = b[0] + pc.dtwi;
        b[3] = b[3] + pc.dtwi;
        b[5] = b[5] + pc.dtwi;
        // A = transpose of the velocity gradient (fenep.f90:541-550), zero
        // velocity beyond the ghost rows of a wall channel
        Lyap3 A;
        {
            const bool rm = !(WALLS && j == 0), rp = !(WALLS && j == g.ny + 1);
            auto at = [&](const double *F, int di, int dj, int dk) {
                if (WALLS && ((dj < 0 && !rm) || (dj > 0 && !rp))) return 0.0;
                return F[h + di * ox + dj * oy + dk * oz];
            };
            A.a00 = u00;
            A.a11 = u11;
            A.a22 = u22;
            A.a10 = div_by(-dt * (-at(V, -1, -1, 0) + at(V, 1, -1, 0) - at(V, -1, 0, 0) + at(V, 1, 0, 0)), pc.d4[0]);
            A.a20 = div_by(-dt * (-at(W, -1, 0, -1) + at(W, 1, 0, -1) - at(W, -1, 0, 0) + at(W, 1, 0, 0)), pc.d4[0]);
            A.a01 = div_by(-dt * (-at(U, -1, -1, 0) - at(U, 0, -1, 0) + at(U, -1, 1, 0) + at(U, 0, 1, 0)), pc.d4[1]);
            A.a21 = div_by(-dt * (-at(W, 0, -1, -1) + at(W, 0, 1, -1) - at(W, 0, -1, 0) + at(W, 0, 1, 0)), pc.d4[1]);
            A.a02 = div_by(-dt * (-at(U, -1, 0, -1) - at(U, 0, 0, -1) + at(U, -1, 0, 1) + at(U, 0, 0, 1)), pc.d4[2]);
            A.a12 = div_by(-dt * (-at(V, 0, -1, -1) - at(V, 0, 0, -1) + at(V, 0, -1, 1) + at(V, 0, 0, 1)), pc.d4[2]);
        }
        int itr;
#pragma unroll 1
        for (itr = 1; itr <= ph.newton_itrmax; ++itr) {
            double Ah[6][7], r[6];
            lyap_system(A, b, x, ph.lp2, dt, ph.newton_dc, pc, Ah);
            if (!gauss_diagonal<6>(Ah, r)) {
                // copies, so that the operands of the usual path stay in registers
                const Lyap3 A2 = A;
                double b2[6], x2[6], r2[6];
#pragma unroll
                for (int m = 0; m < 6; ++m) { b2[m] = b[m]; x2[m] = x[m]; }
                lyap_step_pivoting(A2, b2, x2, ph.lp2, dt, ph.newton_dc, pc, r2);
#pragma unroll
                for (int m = 0; m < 6; ++m) r[m] = r2[m];
            }
#pragma unroll
            for (int m = 0; m < 6; ++m) x[m] = x[m] - r[m];
            double sr = 0, sx = 0;
#pragma unroll
            for (int m = 0; m < 6; ++m) sr = sr + r[m] * r[m];
#pragma unroll
            for (int m = 0; m < 6; ++m) sx = sx + x[m] * x[m];
            if (newton_small(sr, sx, ph.newton_eps, pc)) break;
        }
        my_itr = (unsigned long long)itr;
        my_unconv = itr > ph.newton_itrmax ? 1ull : 0ull;
#pragma unroll
        for (int m = 0; m < 6; ++m) Cn[(size_t)m * cs + h] = x[m];
        fpet[h] = (ph.lp2 - 3) / (ph.lp2 - x[0] - x[3] - x[5]);
    }
    unsigned long long a = my_itr, b2 = my_unconv;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b2 += __shfl_down_sync(0xffffffffu, b2, o);
    }
    if (((threadIdx.x + blockDim.x * threadIdx.y) & 31) == 0) {
        if (a) atomicAdd(&cnt->newton_iters, a);
        if (b2) atomicAdd(&cnt->newton_unconverged, b2);
    }
}

// ---------------------------------------------------------------------------
// Polymer, 2D (fenep_2d.f90:138-393): closed-form 2x2 eigenvalues, the "last
// candidate >= running best" rule, Cstar with 1/4 weights, 3-unknown Newton.

__device__ inline void eig2(const double *a, double &re1, double &re2) {
    double d = (a[0] - a[2]) * (a[0] - a[2]) + 4.0 * (a[1] * a[1]);
    double s = sqrt(d);
    re1 = (a[0] + a[2] + s) * 0.5;
    re2 = (a[0] + a[2] - s) * 0.5;
}

// returns the reference's index (0 = none qualified -> cell value)
__device__ inline int select2(const double *cm, const double *c0, const double *cp) {
    int index = 0; double mintemp = 0.0;
    for (int l = 1; l <= 3; ++l) {
        double pt[3], nt[3], e[4];
        for (int m = 0; m < 3; ++m) {
            pt[m] = face_p(l, cm[m], c0[m], cp[m]);
            nt[m] = face_n(l, cm[m], c0[m], cp[m]);
        }
        eig2(pt, e[0], e[1]);
        eig2(nt, e[2], e[3]);
        double mv = e[0];
        bool found = !isnan(mv);
        for (int q = 1; q < 4; ++q) {
            if (isnan(e[q])) continue;
            if (!found || e[q] < mv) { mv = e[q]; found = true; }
        }
        if (found && mv >= mintemp) { index = l; mintemp = mv; }
    }
    return index;
}

__global__ void k_polymer_codes2(const double *__restrict__ C, uint8_t *__restrict__ codes,
                                 uint8_t *__restrict__ codes_g, Geo g, int cs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + prow0(g);
    if (i > g.nx || j >= prow0(g) + prows(g)) return;
    const int k = 1;
    double c0[3], cm[3], cp[3];
    const int h = hix(g, i, j, k);
    for (int m = 0; m < 3; ++m) c0[m] = C[(size_t)m * cs + h];
    const int off[2] = {1, g.sx};
    int code = 0;
    for (int d = 0; d < 2; ++d) {
        for (int m = 0; m < 3; ++m) {
            if (d == 1 && g.walls) {
                cm[m] = crow(C + (size_t)m * cs, g, i, j - 1, k);
                cp[m] = crow(C + (size_t)m * cs, g, i, j + 1, k);
            } else {
                cm[m] = C[(size_t)m * cs + h - off[d]];
                cp[m] = C[(size_t)m * cs + h + off[d]];
            }
        }
        int idx = select2(cm, c0, cp);   // 0..3; 0 -> cell value (stored as 3 = "4")
        code |= (idx == 0 ? 3 : idx - 1) << (2 * d);
    }
    if (j >= 1 && j <= g.ny) codes[qix(g, i, j, k)] = (uint8_t)code;
    else codes_g[gcix(g, i, j, k)] = (uint8_t)code;
}

__device__ inline void lyap_func2(const double A0[2][2], const double *b, const double *x, double *l, double lp2,
                                  double dt, Recip wi) {
    double A[2][2] = {{A0[0][0], A0[0][1]}, {A0[1][0], A0[1][1]}};
    double fx = (lp2 - 2) / (lp2 - x[0] - x[2]);
    double dd = (1.0 + div_by(fx * dt, wi)) * 0.5;
    A[0][0] = A[0][0] + dd;
    A[1][1] = A[1][1] + dd;
    l[0] = (A[0][0] + A[0][0]) * x[0] + A[0][1] * x[1] + A[0][1] * x[1] - b[0];
    l[1] = A[1][0] * x[0] + (A[1][1] + A[0][0]) * x[1] + A[0][1] * x[2] - b[1];
    l[2] = A[1][0] * x[1] + A[1][0] * x[1] + (A[1][1] + A[1][1]) * x[2] - b[2];
}

__global__ void k_polymer_update2(const double *__restrict__ C, double *__restrict__ Cn, double *__restrict__ fpet,
                                  const uint8_t *__restrict__ codes, const uint8_t *__restrict__ codes_g,
                                  const double *__restrict__ U, const double *__restrict__ V, Geo g, Phys ph, PolyConst pc,
                                  int cs, StepCounters *cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + prow0(g);
    const int k = 1;
    const bool active = i <= g.nx && j < prow0(g) + prows(g);
    unsigned long long my_itr = 0, my_unconv = 0;
    if (active) {
        const int h = hix(g, i, j, k);
        const double dt = ph.dt;
        const int cself = code_at(codes, codes_g, g, i, j, k);
        const int cxm = code_at(codes, codes_g, g, wrapx(g, i - 1), j, k) & 3;
        const int cxp = code_at(codes, codes_g, g, wrapx(g, i + 1), j, k) & 3;
        int jm = j - 1, jp = j + 1;
        if (!g.walls) { jm = wrapy(g, jm); jp = wrapy(g, jp); }
        const int cym = (jm < 0) ? 3 : (code_at(codes, codes_g, g, i, jm, k) >> 2) & 3;
        const int cyp = (jp > g.ny + 1) ? 3 : (code_at(codes, codes_g, g, i, jp, k) >> 2) & 3;
        const int isx = (cself & 3) + 1, isy = ((cself >> 2) & 3) + 1;
        const int hxm = hix(g, wrapx(g, i - 1), j, k), hxp = hix(g, wrapx(g, i + 1), j, k);
        const int ox = 1;
        double u1 = U[hix(g, i - 1, j, k)], u2 = U[h];
        double v1 = crow(V, g, i, j - 1, k), v2 = V[h];
        double s1 = div_by((-u2 + fabs(u2)) * dt, pc.d2[0]);
        double s2 = 1.0 / 4 + div_by((-u2 - fabs(u2)) * dt, pc.d2[0]);
        double s3 = 1.0 / 4 + div_by((u1 - fabs(u1)) * dt, pc.d2[0]);
        double s4 = div_by((u1 + fabs(u1)) * dt, pc.d2[0]);
        double s5 = div_by((-v2 + fabs(v2)) * dt, pc.d2[1]);
        double s6 = 1.0 / 4 + div_by((-v2 - fabs(v2)) * dt, pc.d2[1]);
        double s7 = 1.0 / 4 + div_by((v1 - fabs(v1)) * dt, pc.d2[1]);
        double s8 = div_by((v1 + fabs(v1)) * dt, pc.d2[1]);
        double b[3], x[3];
        for (int m = 0; m < 3; ++m) {
            const double *Cm = C + (size_t)m * cs;
            const double c0 = Cm[h];
            double pxm = face_p(isx, Cm[h - ox], c0, Cm[h + ox]);
            double nxp = face_n(isx, Cm[h - ox], c0, Cm[h + ox]);
            double pxp = face_p(cxp + 1, Cm[hxp - ox], Cm[hxp], Cm[hxp + ox]);
            double nxm = face_n(cxm + 1, Cm[hxm - ox], Cm[hxm], Cm[hxm + ox]);
            double pym, nyp, pyp, nym;
            if (!g.walls) {   // jm, jp wrapped; rows read around them through the halo
                const int hym = hix(g, i, jm, k), hyp = hix(g, i, jp, k), oy = g.sx;
                pym = face_p(isy, Cm[h - oy], c0, Cm[h + oy]);
                nyp = face_n(isy, Cm[h - oy], c0, Cm[h + oy]);
                pyp = face_p(cyp + 1, Cm[hyp - oy], Cm[hyp], Cm[hyp + oy]);
                nym = face_n(cym + 1, Cm[hym - oy], Cm[hym], Cm[hym + oy]);
            } else {          // zero beyond the ghost rows
                const double ym2 = crow(Cm, g, i, j - 2, k), ym1 = crow(Cm, g, i, j - 1, k);
                const double yp1 = crow(Cm, g, i, j + 1, k), yp2 = crow(Cm, g, i, j + 2, k);
                pym = face_p(isy, ym1, c0, yp1);
                nyp = face_n(isy, ym1, c0, yp1);
                pyp = face_p(cyp + 1, c0, yp1, yp2);
                nym = face_n(cym + 1, ym2, ym1, c0);
            }
            b[m] = s3 * pxm + s1 * pxp + s4 * nxm + s2 * nxp + s7 * pym + s5 * pyp + s8 * nym + s6 * nyp;
            x[m] = c0;
        }
        b[0] = b[0] + pc.dtwi;
        b[2] = b[2] + pc.dtwi;
        auto u = [&](int a, int bb) { return crow(U, g, a, bb, k); };
        auto v = [&](int a, int bb) { return crow(V, g, a, bb, k); };
        double A0[2][2];
        A0[0][0] = div_by(-dt * (-u(i - 1, j) + u(i, j)), pc.d1[0]);
        A0[0][1] = div_by(-dt * (-v(i - 1, j - 1) + v(i + 1, j - 1) - v(i - 1, j) + v(i + 1, j)), pc.d4[0]);
        A0[1][0] = div_by(-dt * (-u(i - 1, j - 1) - u(i, j - 1) + u(i - 1, j + 1) + u(i, j + 1)), pc.d4[1]);
        A0[1][1] = div_by(-dt * (-v(i, j - 1) + v(i, j)), pc.d1[1]);
        double AT[2][2] = {{A0[0][0], A0[1][0]}, {A0[0][1], A0[1][1]}};
        const double dc = ph.newton_dc;
        int itr;
        for (itr = 1; itr <= ph.newton_itrmax; ++itr) {
            double Ah[3][4], x1[3], x2[3], l1[3], l2[3], l[3], r[3];
            for (int col = 0; col < 3; ++col) {
                for (int m = 0; m < 3; ++m) { x1[m] = x[m]; x2[m] = x[m]; }
                x1[col] = x1[col] + dc;
                x2[col] = x2[col] - dc;
                lyap_func2(AT, b, x1, l1, ph.lp2, dt, pc.wi);
                lyap_func2(AT, b, x2, l2, ph.lp2, dt, pc.wi);
                for (int row = 0; row < 3; ++row) Ah[row][col] = div_by(l1[row] - l2[row], pc.dc2);
            }
            lyap_func2(AT, b, x, l, ph.lp2, dt, pc.wi);
            for (int row = 0; row < 3; ++row) Ah[row][3] = l[row];
            double Ag[3][4];
            for (int row = 0; row < 3; ++row)
                for (int q = 0; q < 4; ++q) Ag[row][q] = Ah[row][q];
            if (!gauss_diagonal<3>(Ah, r)) gauss<3>(Ag, r);
            for (int m = 0; m < 3; ++m) x[m] = x[m] - r[m];
            double sr = 0, sx = 0;
            for (int m = 0; m < 3; ++m) sr = sr + r[m] * r[m];
            for (int m = 0; m < 3; ++m) sx = sx + x[m] * x[m];
            if (newton_small(sr, sx, ph.newton_eps, pc)) break;
        }
        my_itr = (unsigned long long)itr;
        my_unconv = itr > ph.newton_itrmax ? 1ull : 0ull;
        for (int m = 0; m < 3; ++m) Cn[(size_t)m * cs + h] = x[m];
        fpet[h] = (ph.lp2 - 2) / (ph.lp2 - x[0] - x[2]);
    }
    unsigned long long a = my_itr, b2 = my_unconv;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b2 += __shfl_down_sync(0xffffffffu, b2, o);
    }
    if (((threadIdx.x + blockDim.x * threadIdx.y) & 31) == 0) {
        if (a) atomicAdd(&cnt->newton_iters, a);
        if (b2) atomicAdd(&cnt->newton_unconverged, b2);
    }
}

// ---------------------------------------------------------------------------
// Momentum: polymer_stress (fenep.f90:645-691), convection (694-734), viscous
// (736-770) and the predictor right-hand side: the CN/AB2 Q of fft_navier
// (fenep.f90:1469-1474) or the explicit Ua of ibm_preliminary (1997-2010, plus
// dt*F as in fenep_2d.f90:1678).  The AB2/trapezoid history is rotated in the
// same pass (fenep.f90:1521-1526).
struct MomArgs {
    const double *U, *V, *W, *P, *C, *fpet;
    double *Ax0, *Ay0, *Az0, *Tx0, *Ty0, *Tz0;
    const double *Fx, *Fy, *Fz;
    double *out[3];     // Q (interior) or Ua (halo)
    double *B[3];       // B (interior), IBM only
    int cs;
    int polymer, ab2_first, ibm;
    double coef_t;      // (1-beta)/(Re Wi)
    double vis;         // beta/Re
};

template <int DIM>
__global__ void __launch_bounds__(256) k_momentum(MomArgs a, Geo g, GridRecip kc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    if (i > g.nx || j > g.ny) return;
    const double dt = g.dt;
    const double *U = a.U, *V = a.V, *W = a.W;
    auto u = [&](int x, int y, int z) { return U[hix(g, x, y, z)]; };
    auto v = [&](int x, int y, int z) { return V[hix(g, x, y, z)]; };
    auto w = [&](int x, int y, int z) { return W[hix(g, x, y, z)]; };
    const int o = qix(g, i, j, k);
    const int h = hix(g, i, j, k);
    // polymer stress
    double tx = 0.0, ty = 0.0, tz = 0.0;
    if (a.polymer) {
        const int cs = a.cs;
        const double *C = a.C, *fp = a.fpet;
        if (DIM == 3) {
            const double E[6] = {1.0, 0.0, 0.0, 1.0, 0.0, 1.0};
            auto c0 = [&](int m, int x, int y, int z) {
                int hh = hix(g, x, y, z);
                return fp[hh] * C[(size_t)(m - 1) * cs + hh] - E[m - 1];
            };
            double sx = div_by(-c0(1, i, j, k) + c0(1, i + 1, j, k), kc.d1[0])
                      + div_by(-c0(2, i, j - 1, k) - c0(2, i + 1, j - 1, k) + c0(2, i, j + 1, k) + c0(2, i + 1, j + 1, k), kc.d4[1])
                      + div_by(-c0(3, i, j, k - 1) - c0(3, i + 1, j, k - 1) + c0(3, i, j, k + 1) + c0(3, i + 1, j, k + 1), kc.d4[2]);
            double sy = div_by(-c0(2, i - 1, j, k) + c0(2, i + 1, j, k) - c0(2, i - 1, j + 1, k) + c0(2, i + 1, j + 1, k), kc.d4[0])
                      + div_by(-c0(4, i, j, k) + c0(4, i, j + 1, k), kc.d1[1])
                      + div_by(-c0(5, i, j, k - 1) - c0(5, i, j + 1, k - 1) + c0(5, i, j, k + 1) + c0(5, i, j + 1, k + 1), kc.d4[2]);
            double sz = div_by(-c0(3, i - 1, j, k) + c0(3, i + 1, j, k) - c0(3, i - 1, j, k + 1) + c0(3, i + 1, j, k + 1), kc.d4[0])
                      + div_by(-c0(5, i, j - 1, k) + c0(5, i, j + 1, k) - c0(5, i, j - 1, k + 1) + c0(5, i, j + 1, k + 1), kc.d4[1])
                      + div_by(-c0(6, i, j, k) + c0(6, i, j, k + 1), kc.d1[2]);
            tx = a.coef_t * sx; ty = a.coef_t * sy; tz = a.coef_t * sz;
        } else {
            const double E[3] = {1.0, 0.0, 1.0};
            auto c0 = [&](int m, int x, int y) {
                int hh = hix(g, x, y, k);
                return fp[hh] * C[(size_t)(m - 1) * cs + hh] - E[m - 1];
            };
            double sx = div_by(-c0(1, i, j) + c0(1, i + 1, j), kc.d1[0])
                      + div_by(-c0(2, i, j - 1) - c0(2, i + 1, j - 1) + c0(2, i, j + 1) + c0(2, i + 1, j + 1), kc.d4[1]);
            double sy = div_by(-c0(2, i - 1, j) + c0(2, i + 1, j) - c0(2, i - 1, j + 1) + c0(2, i + 1, j + 1), kc.d4[0])
                      + div_by(-c0(3, i, j) + c0(3, i, j + 1), kc.d1[1]);
            tx = a.coef_t * sx; ty = a.coef_t * sy;
        }
    }
    // convection and viscous terms
    double t1 = (u(i - 1, j, k) + u(i, j, k)) / 2, t2 = (u(i, j, k) + u(i + 1, j, k)) / 2;
    double ax = div_by(-(t1 * t1) + t2 * t2, kc.d1[0])
              + div_by(-(v(i, j - 1, k) + v(i + 1, j - 1, k)) / 2 * (u(i, j - 1, k) + u(i, j, k)) / 2
                 + (v(i, j, k) + v(i + 1, j, k)) / 2 * (u(i, j, k) + u(i, j + 1, k)) / 2, kc.d1[1]);
    double t3 = (v(i, j - 1, k) + v(i, j, k)) / 2, t4 = (v(i, j, k) + v(i, j + 1, k)) / 2;
    double ay = div_by(-(u(i - 1, j, k) + u(i - 1, j + 1, k)) / 2 * (v(i - 1, j, k) + v(i, j, k)) / 2
                 + (u(i, j, k) + u(i, j + 1, k)) / 2 * (v(i, j, k) + v(i + 1, j, k)) / 2, kc.d1[0])
              + div_by(-(t3 * t3) + t4 * t4, kc.d1[1]);
    double bx = div_by(u(i - 1, j, k) - 2 * u(i, j, k) + u(i + 1, j, k), kc.dd[0])
              + div_by(u(i, j - 1, k) - 2 * u(i, j, k) + u(i, j + 1, k), kc.dd[1]);
    double by = div_by(v(i - 1, j, k) - 2 * v(i, j, k) + v(i + 1, j, k), kc.dd[0])
              + div_by(v(i, j - 1, k) - 2 * v(i, j, k) + v(i, j + 1, k), kc.dd[1]);
    double az = 0, bz = 0;
    if (DIM == 3) {
        ax = ax + div_by(-(w(i, j, k - 1) + w(i + 1, j, k - 1)) / 2 * (u(i, j, k - 1) + u(i, j, k)) / 2
                   + (w(i, j, k) + w(i + 1, j, k)) / 2 * (u(i, j, k) + u(i, j, k + 1)) / 2, kc.d1[2]);
        ay = ay + div_by(-(w(i, j, k - 1) + w(i, j + 1, k - 1)) / 2 * (v(i, j, k - 1) + v(i, j, k)) / 2
                   + (w(i, j, k) + w(i, j + 1, k)) / 2 * (v(i, j, k) + v(i, j, k + 1)) / 2, kc.d1[2]);
        double t5 = (w(i, j, k - 1) + w(i, j, k)) / 2, t6 = (w(i, j, k) + w(i, j, k + 1)) / 2;
        az = div_by(-(u(i - 1, j, k) + u(i - 1, j, k + 1)) / 2 * (w(i - 1, j, k) + w(i, j, k)) / 2
              + (u(i, j, k) + u(i, j, k + 1)) / 2 * (w(i, j, k) + w(i + 1, j, k)) / 2, kc.d1[0])
           + div_by(-(v(i, j - 1, k) + v(i, j - 1, k + 1)) / 2 * (w(i, j - 1, k) + w(i, j, k)) / 2
              + (v(i, j, k) + v(i, j, k + 1)) / 2 * (w(i, j, k) + w(i, j + 1, k)) / 2, kc.d1[1])
           + div_by(-(t5 * t5) + t6 * t6, kc.d1[2]);
        bx = bx + div_by(u(i, j, k - 1) - 2 * u(i, j, k) + u(i, j, k + 1), kc.dd[2]);
        by = by + div_by(v(i, j, k - 1) - 2 * v(i, j, k) + v(i, j, k + 1), kc.dd[2]);
        bz = div_by(w(i - 1, j, k) - 2 * w(i, j, k) + w(i + 1, j, k), kc.dd[0])
           + div_by(w(i, j - 1, k) - 2 * w(i, j, k) + w(i, j + 1, k), kc.dd[1])
           + div_by(w(i, j, k - 1) - 2 * w(i, j, k) + w(i, j, k + 1), kc.dd[2]);
    }
    const double A[3] = {-ax, -ay, -az};
    const double B[3] = {a.vis * bx, a.vis * by, a.vis * bz};
    const double T[3] = {tx, ty, tz};
    double *A0p[3] = {a.Ax0, a.Ay0, a.Az0};
    double *T0p[3] = {a.Tx0, a.Ty0, a.Tz0};
    const double *Fp[3] = {a.Fx, a.Fy, a.Fz};
    const double *Us[3] = {U, V, W};
    const int hp[3] = {hix(g, i + 1, j, k), hix(g, i, j + 1, k), hix(g, i, j, k + 1)};
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
        double a0 = a.ab2_first ? A[c] : A0p[c][o];
        double t0 = a.ab2_first ? T[c] : T0p[c][o];
        double gp = div_by(-dt * (-a.P[h] + a.P[hp[c]]), kc.d1[c]);
        double val;
        if (!a.ibm)
            val = Us[c][h] + gp + dt * (3.0 * A[c] - a0) / 2.0 + dt * B[c] / 2.0 + dt * (T[c] + t0) / 2.0 + dt * Fp[c][o];
        else
            val = Us[c][h] + gp + dt * (3.0 * A[c] - a0) / 2.0 + dt * B[c] + dt * (T[c] + t0) / 2.0 + dt * Fp[c][o];
        if (!a.ibm) a.out[c][o] = val;
        else { a.out[c][h] = val; a.B[c][o] = B[c]; }
        A0p[c][o] = A[c];
        T0p[c][o] = T[c];
    }
}

// ---------------------------------------------------------------------------
// IBM (fenep_mpi.f90:1794-1929; 2D fenep_2d.f90:1726-1819).

__device__ inline double roma(double r) {
    double ar = fabs(r);
    if (ar < 1.5 && ar >= 0.5) return (5.0 - 3.0 * ar - sqrt(-3.0 * ((1 - ar) * (1 - ar)) + 1.0)) / 6.0;
    if (ar < 0.5) return (1.0 + sqrt(-3.0 * (r * r) + 1.0)) / 3.0;
    return 0.0;
}

__device__ inline void stencil_origin(int comp, double xc, double yc, double dX, double dY, int &i0, int &j0) {
    if (comp == 0) { j0 = (int)(yc / dY); i0 = (int)(xc / dX - 0.5); }
    else if (comp == 1) { j0 = (int)(yc / dY - 0.5); i0 = (int)(xc / dX); }
    else { j0 = (int)(yc / dY); i0 = (int)(xc / dX); }
}

__device__ inline void grid_pos(int comp, int i, int j, int k, double dX, double dY, double dZ, double &x, double &y,
                                double &z) {
    x = (i - 0.5) * dX; y = (j - 0.5) * dY; z = (k - 0.5) * dZ;
    if (comp == 0) x = x + 0.5 * dX;
    else if (comp == 1) y = y + 0.5 * dY;
    else z = z + 0.5 * dZ;
}

struct IbmArgs {
    const double *mx, *my, *mu, *mv;
    const int *mcyl;
    int nm, ncomp, d3;
    Recip dvol;                // cell volume
    double dxn;
    const double *mvol;        // per marker: spreading volume (dX^3, or the ring's arc element)
    int accumulate;            // forcing iteration > 1: Fc += (Uc - Ub)/dt (smac.f90:1345-1353)
    const double *Uf[3];
    double *Fc[3];
    const int *off[3], *idx[3];
    const double *Ua[3], *B[3];
    double *Q[3];
    // kernel weight tables (k_marker_weights): roma of the x, y offsets of each
    // marker's 3 stencil columns / rows, and of the z offsets of planes n-1..n+1
    const double *wx[3], *wy[3], *wz[3];
    const int *i0[3], *j0[3];
};

// Tables of the Roma weights (fenep.f90:2045-2055): the same expressions as the
// reference's delta evaluation inside its stencil loops, evaluated once per
// marker (x, y) and per plane (z), so that each product below is the same double.
__global__ void k_marker_weights(const double *mx, const double *my, int nm, int comp, Geo g, double *wx, double *wy,
                                 int *i0o, int *j0o) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nm) return;
    const double dX = g.dx, dY = g.dy, dZ = g.dz;
    const double xc = mx[m], yc = my[m];
    int i0, j0;
    stencil_origin(comp, xc, yc, dX, dY, i0, j0);
    i0o[m] = i0;
    j0o[m] = j0;
    for (int a = 0; a < 3; ++a) {
        double x, y, z;
        grid_pos(comp, i0 + a, j0 + a, 1, dX, dY, dZ, x, y, z);
        wx[3 * m + a] = roma((x - xc) / dX);
        wy[3 * m + a] = roma((y - yc) / dY);
    }
}

__global__ void k_plane_weights(int comp, Geo g, double *wz) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (n > g.nz) return;
    const double dX = g.dx, dY = g.dy, dZ = g.dz;
    const double zc = (n - 0.25) * dZ;
    for (int c = 0; c < 3; ++c) {
        double x, y, z;
        grid_pos(comp, 1, 1, n - 1 + c, dX, dY, dZ, x, y, z);
        wz[3 * (n - 1) + c] = roma((z - zc) / dZ);
    }
}

// delta(x_e - X_m) of stencil cell (a, b, c) of marker m on plane n
__device__ inline double ibm_delta(const IbmArgs &a, int comp, int m, int n, int ia, int jb, int kc) {
    const double xy = a.wx[comp][3 * m + ia] * a.wy[comp][3 * m + jb];
    return div_by(a.d3 ? xy * a.wz[comp][3 * (n - 1) + kc] : xy, a.dvol);
}

// interpolation at the markers and the marker force Fc = (Uc - Ub)/dt
__global__ void k_ibm_interp(IbmArgs a, Geo g) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = blockIdx.y + 1;
    const int comp = blockIdx.z;
    if (m >= a.nm) return;
    const int i0 = a.i0[comp][m], j0 = a.j0[comp][m];
    const int klo = a.d3 ? n - 1 : 1, khi = a.d3 ? n + 1 : 1;
    double ub = 0.0;
    const double *Uf = a.Uf[comp];
    for (int k = klo; k <= khi; ++k)
        for (int j = j0; j <= j0 + 2; ++j)
            for (int i = i0; i <= i0 + 2; ++i) {
                const double del = ibm_delta(a, comp, m, n, i - i0, j - j0, k - klo);
                ub = ub + Uf[hix(g, i, j, k)] * del * a.dxn;
            }
    const double uc = comp == 0 ? a.mu[m] : (comp == 1 ? a.mv[m] : 0.0);
    double *fc = &a.Fc[comp][m + (size_t)a.nm * (n - 1)];
    *fc = (a.accumulate ? *fc : 0.0) + (uc - ub) / g.dt;
}

// pre-fold spreading sum of extended cell (ie, je, ke) (ftmp of ibm_Helmholtz)
__device__ inline double spread_at(const IbmArgs &a, const Geo &g, int comp, int ie, int je, int ke) {
    const int col = ie + g.sx * je;
    const int b = a.off[comp][col], e = a.off[comp][col + 1];
    if (b == e) return 0.0;
    double acc = 0.0;
    const int nlo = a.d3 ? max(ke - 1, 1) : 1, nhi = a.d3 ? min(ke + 1, g.nz) : 1;
    for (int n = nlo; n <= nhi; ++n) {
        const int kc = a.d3 ? ke - n + 1 : 0;
        for (int q = b; q < e; ++q) {
            const int m = a.idx[comp][q];
            const double del = ibm_delta(a, comp, m, n, ie - a.i0[comp][m], je - a.j0[comp][m], kc);
            double fcv = a.Fc[comp][m + (size_t)a.nm * (n - 1)];
            acc = acc + fcv * del * a.mvol[m];
        }
    }
    return acc;
}

// Spread the marker forces (with the periodic fold of ibm_PBM,
// fenep.f90:2195-2205) and form Q = Ua + dt*f - dt*B/2 (ibm_predict,
// fenep.f90:2229) for every interior cell; a thread per cell and component (the
// few cells under a cylinder sum tens of entries each, in a serial FP64 chain).
__global__ void k_ibm_spread_q(IbmArgs a, Geo g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int comp = blockIdx.z / g.nz, k = blockIdx.z - comp * g.nz + 1;
    if (i > g.nx || j > g.ny) return;
    const int o = qix(g, i, j, k), h = hix(g, i, j, k);
    int xs[2] = {i, -1}, ys[2] = {j, -1}, zs[2] = {k, -1};
    if (i == 1) xs[1] = g.nx + 1; else if (i == g.nx) xs[1] = 0;
    if (!g.walls) { if (j == 1) ys[1] = g.ny + 1; else if (j == g.ny) ys[1] = 0; }
    if (a.d3) { if (k == 1) zs[1] = g.nz + 1; else if (k == g.nz) zs[1] = 0; }
    double fz = 0.0;
    for (int zz = 0; zz < 2; ++zz) {
        if (zs[zz] < 0) continue;
        double fy = 0.0;
        for (int yy = 0; yy < 2; ++yy) {
            if (ys[yy] < 0) continue;
            double fx = 0.0;
            for (int xx = 0; xx < 2; ++xx) {
                if (xs[xx] < 0) continue;
                double v = spread_at(a, g, comp, xs[xx], ys[yy], zs[zz]);
                fx = xx == 0 ? v : fx + v;
            }
            fy = yy == 0 ? fx : fy + fx;
        }
        fz = zz == 0 ? fy : fz + fy;
    }
    const double dt = g.dt;
    a.Q[comp][o] = a.Ua[comp][h] + dt * fz - dt * a.B[comp][o] / 2;
}

// drag of each cylinder: -sum(Fc) * dv per component.  Block (l, n) sums the
// forces of cylinder l's markers on plane n (markers listed per cylinder in
// mperm, ranges moff); the cylinder's last block to finish sums the planes.
// Fixed tree orders make the result deterministic.  A thread's markers are
// summed in their order with the loads of U of them ahead: one at a time, the
// chain of list, force and sum over the 5344 markers of a 512^2 box took 24.5 us,
// with U = 8 14.8 us.  Where a cylinder has no more than two per thread, U = 1
// leaves the side stream's neighbours more of the SM.
__device__ inline void drag_tree(double (&sh)[3][256], const double (&s)[3]) {
    for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] = s[c];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] += sh[c][threadIdx.x + w];
        __syncthreads();
    }
}

template <int U>
__global__ void __launch_bounds__(256) k_drag(const double *Fx, const double *Fy, const double *Fz, const int *mperm,
                                              const int *moff, int nm, int ncomp, double *part, unsigned *done,
                                              const double *cylvol, double *out) {
    const int l = blockIdx.x, n = blockIdx.y, nz = gridDim.y;
    __shared__ double sh[3][256];
    __shared__ bool last;
    double s[3] = {0.0, 0.0, 0.0};
    const double *F[3] = {Fx, Fy, Fz};
    const int end = moff[l + 1];
    for (int q0 = moff[l] + threadIdx.x; q0 < end; q0 += U * 256) {
        int m[U];
        double v[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u) m[u] = q0 + 256 * u < end ? mperm[q0 + 256 * u] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[u][c] = m[u] >= 0 && c < ncomp ? F[c][(size_t)m[u] + (size_t)nm * n] : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (m[u] >= 0)
#pragma unroll
                for (int c = 0; c < 3; ++c) s[c] += v[u][c];
    }
    drag_tree(sh, s);
    if (threadIdx.x == 0) {
        for (int c = 0; c < 3; ++c) part[((size_t)l * nz + n) * 3 + c] = sh[c][0];
        __threadfence();
        last = atomicInc(&done[l], nz - 1) == (unsigned)(nz - 1);   // wraps to 0 for the next launch
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    for (int c = 0; c < 3; ++c) s[c] = 0.0;
    for (int p = threadIdx.x; p < nz; p += blockDim.x)
        for (int c = 0; c < 3; ++c) s[c] += __ldcg(&part[((size_t)l * nz + p) * 3 + c]);
    drag_tree(sh, s);
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; ++c) out[3 * l + c] = c < ncomp ? -sh[c][0] * cylvol[l] : 0.0;
}

// ---------------------------------------------------------------------------
// Poisson right-hand side (fenep.f90:1547-1555) and projection (1562-1604).

__global__ void k_poisson_rhs(const double *Up, const double *Vp, const double *Wp, double *Q, Geo g, GridRecip kc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    if (i > g.nx || j > g.ny) return;
    double s = div_by(-Up[hix(g, i - 1, j, k)] + Up[hix(g, i, j, k)], kc.d1[0]) + div_by(-Vp[hix(g, i, j - 1, k)] + Vp[hix(g, i, j, k)], kc.d1[1]);
    if (g.dim == 3) s = s + div_by(-Wp[hix(g, i, j, k - 1)] + Wp[hix(g, i, j, k)], kc.d1[2]);
    Q[qix(g, i, j, k)] = div_by(s, kc.dt);
}

__global__ void k_march(double *U, double *V, double *W, double *P, const double *Up, const double *Vp,
                        const double *Wp, const double *Phi, Geo g, GridRecip kc, double pc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    if (i > g.nx || j > g.ny) return;
    const int h = hix(g, i, j, k);
    const double dt = g.dt;
    const double ph = Phi[h];
    U[h] = Up[h] - div_by(dt * (-ph + Phi[hix(g, i + 1, j, k)]), kc.d1[0]);
    V[h] = Vp[h] - div_by(dt * (-ph + Phi[hix(g, i, j + 1, k)]), kc.d1[1]);
    if (g.dim == 3) W[h] = Wp[h] - div_by(dt * (-ph + Phi[hix(g, i, j, k + 1)]), kc.d1[2]);
    double lap = div_by(Phi[hix(g, i - 1, j, k)] - 2 * ph + Phi[hix(g, i + 1, j, k)], kc.dd[0])
               + div_by(Phi[hix(g, i, j - 1, k)] - 2 * ph + Phi[hix(g, i, j + 1, k)], kc.dd[1]);
    if (g.dim == 3) lap = lap + div_by(Phi[hix(g, i, j, k - 1)] - 2 * ph + Phi[hix(g, i, j, k + 1)], kc.dd[2]);
    P[h] = P[h] + ph - pc * lap;
}

// ---------------------------------------------------------------------------
// Reductions.  The red-black SOR itself is in f8_sor.cuh (the reference's
// sweep, fenep.f90:885-896, is lexicographic in k and j; the GPU colours by
// (i+j+k) parity, so it matches the reference only at the converged tolerance).

// Deterministic two-level reductions: partial sums per block in a fixed order,
// then one block sums the partials.
template <int OP>  // 0: sum of squares, 1: sum of interior values of a halo field, 2: sum of values
__global__ void k_reduce_part(const double *A, int n, double *part, Geo g) {
    __shared__ double sh[256];
    double s = 0.0;
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
        if (OP == 0) { double v = A[q]; s += v * v; }
        else if (OP == 2) s += A[q];
        else {
            int i = 1 + (int)(q % g.nx), j = 1 + (int)((q / g.nx) % g.ny), k = 1 + (int)(q / ((long)g.nx * g.ny));
            s += A[hix(g, i, j, k)];
        }
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// finish: scal[slot] = sum(part), with the reference's guard for a zero sum
// when it becomes the SOR's er0
__global__ void k_reduce_final(const double *part, int nparts, double *scal, int slot, int guard) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int q = threadIdx.x; q < nparts; q += blockDim.x) s += part[q];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) scal[slot] = guard && sh[0] == 0.0 ? 1.0e-16 : sh[0];
}

__global__ void k_shift(double *A, int n, const double *scal, int slot, double inv_n) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    double mean = scal[slot] * inv_n;
    A[q] = A[q] - mean;
}

__global__ void k_aos_to_soa(const double *aos, double *soa, int ncomp, int cs) {
    int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= cs) return;
    for (int m = 0; m < ncomp; ++m) soa[(size_t)m * cs + h] = aos[(size_t)ncomp * h + m];
}
__global__ void k_soa_to_aos(const double *soa, double *aos, int ncomp, int cs) {
    int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= cs) return;
    for (int m = 0; m < ncomp; ++m) aos[(size_t)ncomp * h + m] = soa[(size_t)m * cs + h];
}
__global__ void k_count_nonfinite(const double *a, int n, unsigned long long *out) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long c = (q < n && !isfinite(a[q])) ? 1ull : 0ull;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ---------------------------------------------------------------------------
// host helpers

inline dim3 cell_grid(const Geo &g, dim3 blk) {
    return dim3((g.nx + blk.x - 1) / blk.x, (g.ny + blk.y - 1) / blk.y, g.nz);
}

cudaError_t bc_set(const Geo &g, int n, double *const *A, const int *kind, cudaStream_t s) {
    BcSetD b{};
    b.n = n;
    bool v = false;
    for (int f = 0; f < n; ++f) {
        b.A[f] = A[f];
        b.kind[f] = kind[f];
        v = v || kind[f] == BC_V;
    }
    const long t = halo_count(g) + (v && g.walls ? (long)g.nx * g.nz : 0);
    k_bc_set64<<<(unsigned)((t + 255) / 256), 256, 0, s>>>(b, g); count_launch();
    return cudaGetLastError();
}

cudaError_t bc(double *A, const Geo &g, int kind, cudaStream_t s) { return bc_set(g, 1, &A, &kind, s); }

// U, V, (W,) P
cudaError_t bc_state(Dev &d, cudaStream_t s) {
    double *A3[4] = {d.U, d.V, d.W, d.P}, *A2[3] = {d.U, d.V, d.P};
    const int k3[4] = {BC_U, BC_V, BC_W, BC_P}, k2[3] = {BC_U, BC_V, BC_P};
    return d.g.dim == 3 ? bc_set(d.g, 4, A3, k3, s) : bc_set(d.g, 3, A2, k2, s);
}

// The spectral solves of nb systems (interior right-hand sides -> halo fields)
// in one launch per pass: periodic (fft_solve), or with walls FFT(x, z) of rows
// 1..NY, the tridiagonal systems in y over rows 0..NY+1 and the inverse FFT of
// all NY+2 rows.  sys: 0 U/W, 1 V, 2 P; top: the top ghost value of mode (0, 0).
cudaError_t solve_batch(Dev &d, int nb, const double *const *src, double *const *dst, const int *sys, const double *top,
                        cudaStream_t s) {
    const Geo &g = d.g;
    Batch<const double *> in{};
    Batch<XOutD> out{};
    Batch<WallItem<double>> items{};
    for (int q = 0; q < nb; ++q) {
        in.p[q] = src[q];
        out.p[q] = XOutD{dst[q]};
        items.p[q] = WallItem<double>{sys[q], d.walltab[sys[q]], top[q]};
    }
    if (!g.walls) {
        const bool p = sys[0] == SYS_P;
        fft_solve_passes<double, double, XOutD>(nb, in, d.H, d.nspec, out, g.nx, g.ny, g.nz, 1, g.sx, g.sy, 0, d.twx_r,
                                                d.twx_i, d.twy_r, d.twy_i, d.twz_r, d.twz_i, d.kx2, d.ky2, d.kz2,
                                                p ? 0.0 : 1.0, p ? -1.0 : d.ph.dt * d.ph.beta / d.ph.re / 2.0, s);
    } else {
        wall_solve_passes<double, double, XOutD>(nb, in, d.H, d.nspec, out, g, d.twx_r, d.twx_i, d.twz_r, d.twz_i,
                                                 wall_spec(g, d.ph, d.kx2, d.kz2), items, s);
    }
    return cudaGetLastError();
}

cudaError_t solve_one(Dev &d, const double *src, double *dst, int sys, cudaStream_t s) {
    const double top = 0.0;
    return solve_batch(d, 1, &src, &dst, &sys, &top, s);
}

// Red-black SOR (f8_sor.cuh; the reference's poisson, fenep.f90:848-905) of the
// right-hand side Q (interior) into the halo field Phi, which holds the start
// value.  Stops when sqrt(sum E^2 / sum Q^2) < eps, E the residuals of a sweep,
// or after itrmax sweeps (*iters = itrmax + 1), then shifts Phi to zero mean
// (fenep_2d.f90:577-579).
cudaError_t sor_solve_on(Dev &d, const double *Q, double *Phi, double omega, double eps, int itrmax, int *iters,
                         cudaStream_t s) {
    const Geo &g = d.g;
    const int nb = std::min(1024, (d.ni + 255) / 256);
    // er0 = sum(Q^2) (+1e-16 guard)
    k_reduce_part<0><<<nb, 256, 0, s>>>(Q, d.ni, d.red, g); count_launch();
    k_reduce_final<<<1, 256, 0, s>>>(d.red, nb, d.scal, 0, 1); count_launch();
    SorArgs<double> a{};
    a.Phi = Phi; a.R = Q; a.er0 = d.scal; a.part = reinterpret_cast<SorSum<double> *>(d.red); a.flag = d.flag;
    a.om = omega;
    a.bx = 1.0 / (g.dx * g.dx); a.by = 1.0 / (g.dy * g.dy); a.bz = g.dim == 3 ? 1.0 / (g.dz * g.dz) : 0.0;
    a.b0 = a.bx + a.bx + a.by + a.by + a.bz + a.bz;
    a.rb0 = recip(a.b0);
    a.eps = eps; a.itrmax = itrmax;
    F8_CUDA_RET(sor_sweeps(a, g, device_sm_count(), 1, s));
    int it_host[3] = {0, 0, 0};
    F8_CUDA_RET(cudaMemcpyAsync(it_host, d.flag, sizeof(it_host), cudaMemcpyDeviceToHost, s));
    F8_CUDA_RET(cudaStreamSynchronize(s));
    if (it_host[2]) return cudaErrorTimeout;      // a wait of the grid barrier ran out
    *iters = it_host[0] ? it_host[1] : itrmax + 1;
    F8_CUDA_RET(bc(Phi, g, BC_P, s));
    // zero-mean shift (fenep_2d.f90:577-579)
    k_reduce_part<1><<<nb, 256, 0, s>>>(Phi, d.ni, d.red, g); count_launch();
    k_reduce_final<<<1, 256, 0, s>>>(d.red, nb, d.scal, 2, 0); count_launch();
    k_shift<<<(d.cs + 255) / 256, 256, 0, s>>>(Phi, d.cs, d.scal, 2, 1.0 / ((double)g.nx * g.ny * g.nz)); count_launch();
    return cudaGetLastError();
}

cudaError_t sor_solve(Dev &d, const StepOpts &o, int *iters, cudaStream_t s) {
    return sor_solve_on(d, d.Q[0], d.Phi, o.sor_omega, o.sor_eps, o.sor_itrmax, iters, s);
}

// subtract the mean of an interior field (n values)
cudaError_t remove_mean(Dev &d, double *A, int n, cudaStream_t s) {
    int nb = std::min(1024, (n + 255) / 256);
    k_reduce_part<2><<<nb, 256, 0, s>>>(A, n, d.red, d.g); count_launch();
    k_reduce_final<<<1, 256, 0, s>>>(d.red, nb, d.scal, 3, 0); count_launch();
    k_shift<<<(n + 255) / 256, 256, 0, s>>>(A, n, d.scal, 3, 1.0 / n); count_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t init_kernels_fp64() {
    const int big = 200 * 1024;
    F8_CUDA_RET(cudaFuncSetAttribute(k_fft_lines<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    F8_CUDA_RET(cudaFuncSetAttribute(k_fft_x_fwd<double, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    F8_CUDA_RET(cudaFuncSetAttribute(k_fft_x_inv<double, XOutD>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    return cudaSuccess;
}

cudaError_t bc_all_state_fp64(Dev &d, cudaStream_t s) {
    cudaError_t e;
    if ((e = bc_state(d, s))) return e;
    long n = halo_count(d.g);
    k_bc_c_pet<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d.C, d.fpet, d.g, d.ncomp, d.cs, d.ph.lp2); count_launch();
    k_pet_all<<<(d.cs + 255) / 256, 256, 0, s>>>(d.C, d.fpet, d.ncomp, d.cs, d.ph.lp2); count_launch();
    return cudaGetLastError();
}

cudaError_t bc_field(double *A, const Geo &g, int kind, cudaStream_t s) { return bc(A, g, kind, s); }

cudaError_t helmholtz_solves_fp64(Dev &d, int ncomp, const double *const *src, double *const *dst, cudaStream_t s) {
    const int sys[3] = {SYS_U, SYS_V, SYS_U};
    const double top[3] = {0.0, 0.0, 0.0};
    return solve_batch(d, ncomp, src, dst, sys, top, s);
}

cudaError_t sor_solve_fp64(Dev &d, const double *Q, double *Phi, double omega, double eps, int itrmax, int *iters,
                           cudaStream_t s) {
    return sor_solve_on(d, Q, Phi, omega, eps, itrmax, iters, s);
}

cudaError_t remove_mean_fp64(Dev &d, double *A, int n, cudaStream_t s) { return remove_mean(d, A, n, s); }

cudaError_t poisson_solve_fp64(Dev &d, const double *src, double *dst, cudaStream_t s) {
    return solve_one(d, src, dst, SYS_P, s);
}

cudaError_t wall_tables_fp64(Dev &d, cudaStream_t s) {
    const Geo &g = d.g;
    for (int sys = 0; sys < 3; ++sys)
        wall_table<double>(d.walltab[sys], g.ny, g.nx / 2 + 1, g.nz, wall_spec(g, d.ph, d.kx2, d.kz2), sys, s);
    return cudaGetLastError();
}

cudaError_t launch_poisson_rhs(Dev &d, double *out, cudaStream_t s) {
    dim3 blk(32, 8);
    k_poisson_rhs<<<cell_grid(d.g, blk), blk, 0, s>>>(d.Up, d.Vp, d.Wp, out, d.g, grid_recip(d.g)); count_launch();
    return cudaGetLastError();
}

cudaError_t launch_march(Dev &d, cudaStream_t s) {
    dim3 blk(32, 8);
    k_march<<<cell_grid(d.g, blk), blk, 0, s>>>(d.U, d.V, d.W, d.P, d.Up, d.Vp, d.Wp, d.Phi, d.g, grid_recip(d.g),
                                                d.ph.dt * d.ph.beta / d.ph.re / 2.0); count_launch();
    return cudaGetLastError();
}

cudaError_t marker_weights_fp64(Dev &d, cudaStream_t s) {
    const int ncomp = d.g.dim == 3 ? 3 : 2;
    for (int c = 0; c < ncomp; ++c) {
        k_marker_weights<<<(d.nm + 127) / 128, 128, 0, s>>>(d.mx, d.my, d.nm, c, d.g, d.mwxd[c], d.mwyd[c], d.mi0d[c],
                                                            d.mj0d[c]); count_launch();
        k_plane_weights<<<(d.g.nz + 127) / 128, 128, 0, s>>>(c, d.g, d.mwzd[c]); count_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_drag(Dev &d, double *out, cudaStream_t s) {
    const Geo &g = d.g;
    const bool d3 = g.dim == 3;
    auto go = [&](auto kernel) {
        kernel<<<dim3(d.ncyl, g.nz), 256, 0, s>>>(d.Fc[0], d.Fc[1], d.Fc[2], d.mperm, d.moff, d.nm, d3 ? 3 : 2,
                                                  d.dragpart, d.dragcnt, d.cylvol, out);
    };
    if (d.nm > 512 * d.ncyl) go(k_drag<8>);
    else go(k_drag<1>);
    count_launch();
    return cudaGetLastError();
}

cudaError_t aos_to_soa(const double *aos, double *soa, int ncomp, int cs, cudaStream_t s) {
    k_aos_to_soa<<<(cs + 255) / 256, 256, 0, s>>>(aos, soa, ncomp, cs); count_launch();
    return cudaGetLastError();
}
cudaError_t soa_to_aos(const double *soa, double *aos, int ncomp, int cs, cudaStream_t s) {
    k_soa_to_aos<<<(cs + 255) / 256, 256, 0, s>>>(soa, aos, ncomp, cs); count_launch();
    return cudaGetLastError();
}
cudaError_t count_nonfinite(const double *a, int n, unsigned long long *out, cudaStream_t s) {
    k_count_nonfinite<<<(n + 255) / 256, 256, 0, s>>>(a, n, out); count_launch();
    return cudaGetLastError();
}

// the face candidates of d.C: the filter, then the FP64 test of its queue
static cudaError_t choose_codes3(Dev &d, cudaStream_t s) {
    const Geo &g = d.g;
    F8_CUDA_RET(codes3_filter(d, s));
    // at most two lanes for each (cell, direction); grid-stride beyond the chip
    const long most = 2L * 3 * g.nx * prows(g) * g.nz;
    const unsigned nb = (unsigned)std::min((most + 127) / 128, 16L * device_sm_count());
    k_codes3_exact<<<nb, 128, 0, s>>>(d.C, d.codes, d.codes_g, g, d.cs, codes3_queue(d, 0), codes3_queue(d, 1),
                                      codes3_queue(d, 2), d.code_count); count_launch();
    return cudaGetLastError();
}

cudaError_t step_fp64(Dev &d, const StepOpts &o, double *drag_out_dev, int *sor_iters, cudaStream_t s) {
    const Geo &g = d.g;
    const bool d3 = g.dim == 3;
    cudaError_t e;
    auto mark = [&](int q) { if (o.ev) cudaEventRecord(o.ev[q], s); };
    mark(0);
    // 1. polymer
    if (o.polymer) {
        dim3 blk(32, 4);
        // the rows of the polymer update (with walls the ghost rows too)
        dim3 grd((g.nx + blk.x - 1) / blk.x, (prows(g) + blk.y - 1) / blk.y, g.nz);
        if (o.codes_ready) {
            F8_CUDA_RET(cudaStreamWaitEvent(s, d.ev_code[1], 0));
        } else if (d3 && d.ph.eigen_test == 0) {
            F8_CUDA_RET(choose_codes3(d, s));
        } else if (d3) { k_polymer_codes3<<<grd, blk, 0, s>>>(d.C, d.codes, d.codes_g, g, d.cs, d.ph.eigen_test); count_launch(); }
        else { k_polymer_codes2<<<grd, blk, 0, s>>>(d.C, d.codes, d.codes_g, g, d.cs); count_launch(); }
        mark(1);
        const PolyConst pc = poly_const(g, d.ph);
        if (d3) {
            auto update = g.walls ? k_polymer_update3<true> : k_polymer_update3<false>;
            update<<<grd, blk, 0, s>>>(d.C, d.Cn, d.fpet, d.codes, d.codes_g, d.U, d.V, d.W, g, d.ph, pc, d.cs, d.cnt); count_launch();
        } else { k_polymer_update2<<<grd, blk, 0, s>>>(d.C, d.Cn, d.fpet, d.codes, d.codes_g, d.U, d.V, g, d.ph, pc, d.cs, d.cnt); count_launch(); }
        std::swap(d.C, d.Cn);
        long n = halo_count(g);
        if (g.walls) { k_bc_c_pet_xz<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d.C, d.fpet, g, d.ncomp, d.cs, d.ph.lp2); count_launch(); }
        else { k_bc_c_pet<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d.C, d.fpet, g, d.ncomp, d.cs, d.ph.lp2); count_launch(); }
        if ((e = cudaGetLastError())) return e;
    } else {
        mark(1);
    }
    mark(2);
    // 2. momentum right-hand side
    MomArgs ma{};
    ma.U = d.U; ma.V = d.V; ma.W = d.W; ma.P = d.P; ma.C = d.C; ma.fpet = d.fpet;
    ma.Ax0 = d.Ax0; ma.Ay0 = d.Ay0; ma.Az0 = d.Az0; ma.Tx0 = d.Tx0; ma.Ty0 = d.Ty0; ma.Tz0 = d.Tz0;
    ma.Fx = d.Fx; ma.Fy = d.Fy; ma.Fz = d.Fz;
    if (o.ibm) { ma.out[0] = d.Ua; ma.out[1] = d.Va; ma.out[2] = d.Wa; }
    else { ma.out[0] = d.Q[0]; ma.out[1] = d.Q[1]; ma.out[2] = d.Q[2]; }
    ma.B[0] = d.Bx; ma.B[1] = d.By; ma.B[2] = d.Bz;
    ma.cs = d.cs; ma.polymer = o.polymer; ma.ab2_first = o.ab2_first; ma.ibm = o.ibm;
    ma.coef_t = (1.0 - d.ph.beta) / (d.ph.re * d.ph.wi);
    ma.vis = d.ph.beta / d.ph.re;
    {
        dim3 blk(32, 8);
        dim3 grd = cell_grid(g, blk);
        if (d3) { k_momentum<3><<<grd, blk, 0, s>>>(ma, g, grid_recip(g)); count_launch(); }
        else { k_momentum<2><<<grd, blk, 0, s>>>(ma, g, grid_recip(g)); count_launch(); }
        if ((e = cudaGetLastError())) return e;
    }
    // C is final but for the ghost rows that the momentum stage was the last to
    // read: the next step's face candidates (FP32 but for their queue) beside
    // the FP64 solves.  Six steps of a 64^3 box 12.82 ms with the candidates at the
    // start of each, 12.49 beside; nine of 32x16x16 3.06 and 2.70.
    auto extrapolate = [&](cudaStream_t q) {
        // the wall extrapolation of the ghost rows (C_kabe at the end of the
        // step, fenep_2d.f90:1374)
        k_bc_c_pet<<<(unsigned)((halo_count(g) + 255) / 256), 256, 0, q>>>(d.C, d.fpet, g, d.ncomp, d.cs, d.ph.lp2);
        count_launch();
    };
    if (o.codes_next) {
        F8_CUDA_RET(cudaEventRecord(d.ev_code[0], s));
        F8_CUDA_RET(cudaStreamWaitEvent(d.code_side, d.ev_code[0], 0));
        if (g.walls) extrapolate(d.code_side);
        F8_CUDA_RET(choose_codes3(d, d.code_side));
        F8_CUDA_RET(cudaEventRecord(d.ev_code[1], d.code_side));
    }
    mark(3);
    // 3. IBM direct forcing and 4. Helmholtz (CN viscous) solves; with NS > 1
    // forcing iterations (smac.f90:1607-1611) each further iteration
    // interpolates from the last Helmholtz solution, adds to the marker
    // forces, spreads them and solves again
    double *outs[3] = {d.Up, d.Vp, d.Wp}, *ua[3] = {d.Ua, d.Va, d.Wa};
    const int nv = d3 ? 3 : 2, kinds[3] = {BC_U, BC_V, BC_W};
    IbmArgs ia{};
    if (o.ibm) {
        if ((e = bc_set(g, nv, ua, kinds, s))) return e;
        ia.mx = d.mx; ia.my = d.my; ia.mu = d.mu; ia.mv = d.mv; ia.mcyl = d.mcyl;
        ia.nm = d.nm; ia.ncomp = d3 ? 3 : 2; ia.d3 = d3;
        ia.dvol = recip(d3 ? (g.dx * g.dy) * g.dz : g.dx * g.dy);
        ia.dxn = d3 ? g.dx * g.dx * g.dx : g.dx * g.dx;
        ia.mvol = d.mvol;
        for (int c = 0; c < 3; ++c) {
            ia.Fc[c] = d.Fc[c]; ia.off[c] = d.csr_off[c]; ia.idx[c] = d.csr_idx[c];
            ia.Q[c] = d.Q[c]; ia.B[c] = (c == 0 ? d.Bx : c == 1 ? d.By : d.Bz);
        }
        ia.Ua[0] = d.Ua; ia.Ua[1] = d.Va; ia.Ua[2] = d.Wa;
        for (int c = 0; c < 3; ++c) {
            ia.wx[c] = d.mwxd[c]; ia.wy[c] = d.mwyd[c]; ia.wz[c] = d.mwzd[c];
            ia.i0[c] = d.mi0d[c]; ia.j0[c] = d.mj0d[c];
        }
    }
    const int repeats = o.ibm ? std::max(1, d.ibm_repeats) : 1;
    for (int r = 0; r < repeats; ++r) {
        if (o.ibm) {
            // the first iteration interpolates Ua (Up = Ua, ibm_preliminary)
            const double *src[3] = {d.Ua, d.Va, d.Wa}, *srcp[3] = {d.Up, d.Vp, d.Wp};
            for (int c = 0; c < 3; ++c) ia.Uf[c] = r == 0 ? src[c] : srcp[c];
            ia.accumulate = r > 0;
            dim3 gi((d.nm + 127) / 128, g.nz, ia.ncomp);
            k_ibm_interp<<<gi, 128, 0, s>>>(ia, g); count_launch();
            dim3 blk(32, 8);
            dim3 gs = cell_grid(g, blk);
            gs.z *= ia.ncomp;
            k_ibm_spread_q<<<gs, blk, 0, s>>>(ia, g); count_launch();
            if (r == repeats - 1 && drag_out_dev) F8_CUDA_RET(launch_drag(d, drag_out_dev, s));
            if ((e = cudaGetLastError())) return e;
        }
        if (r == 0) mark(4);
        const int sys[3] = {SYS_U, SYS_V, SYS_U};
        const double top[3] = {2 * g.uwall, 0.0, 0.0};
        if ((e = solve_batch(d, nv, d.Q, outs, sys, top, s))) return e;
        if ((e = bc_set(g, nv, outs, kinds, s))) return e;
    }
    mark(5);
    // 5. Poisson
    {
        dim3 blk(32, 8);
        k_poisson_rhs<<<cell_grid(g, blk), blk, 0, s>>>(d.Up, d.Vp, d.Wp, d.Q[0], g, grid_recip(g)); count_launch();
    }
    if (o.poisson == 0) {
        if ((e = solve_one(d, d.Q[0], d.Phi, SYS_P, s))) return e;
        if ((e = bc(d.Phi, g, BC_P, s))) return e;
        *sor_iters = -1;
    } else {
        if ((e = sor_solve(d, o, sor_iters, s))) return e;
    }
    mark(6);
    // 6. projection and pressure update
    {
        dim3 blk(32, 8);
        k_march<<<cell_grid(g, blk), blk, 0, s>>>(d.U, d.V, d.W, d.P, d.Up, d.Vp, d.Wp, d.Phi, g, grid_recip(g),
                                                  d.ph.dt * d.ph.beta / d.ph.re / 2.0); count_launch();
        if ((e = cudaGetLastError())) return e;
    }
    if ((e = bc_state(d, s))) return e;
    if (o.c_mid) F8_CUDA_RET(cudaMemcpyAsync(o.c_mid, d.C, (size_t)d.ncomp * d.cs * sizeof(double),
                                             cudaMemcpyDeviceToDevice, s));
    if (o.polymer && g.walls && !o.codes_next) extrapolate(s);
    mark(7);
    return cudaGetLastError();
}

}  // namespace f8
