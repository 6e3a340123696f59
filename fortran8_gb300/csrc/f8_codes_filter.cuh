// f8_codes_filter.cuh — the double-float evaluation of the SPD face-candidate
// choice (CpxCnx .. CpzCnz, fenep.f90:169-242) with its error bounds, used by
// k_codes3_filter (f8_codes_fp64.cu, where the bounds are derived).
#pragma once
#include "f8_df64.cuh"

namespace f8 {
namespace codes {

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ df2 dup(df a) { return df2{f2(a.hi), f2(a.lo)}; }
__device__ __forceinline__ df2 scale(df2 a, float w) { return df2{__fmul2_rn(a.hi, f2(w)), __fmul2_rn(a.lo, f2(w))}; }

// 2t(u), u = sqrt(1 - r): the polynomial of the mixed step's eigen test
__device__ __forceinline__ float2 two_t(float2 u) {
    float2 p = f2(-1.993398037e-04f);
    p = __ffma2_rn(p, u, f2(1.522336388e-03f));
    p = __ffma2_rn(p, u, f2(-5.673570558e-03f));
    p = __ffma2_rn(p, u, f2(1.511769835e-02f));
    p = __ffma2_rn(p, u, f2(-3.736452013e-02f));
    p = __ffma2_rn(p, u, f2(1.110385135e-01f));
    p = __ffma2_rn(p, u, f2(-8.164918423e-01f));
    return __ffma2_rn(p, u, f2(-1.0f));
}

// one face from p (times 6), det(B), 1 - r^2 (times p^3, scaled) in FP32:
// lambda - m0 and its bound; false when the face has to be evaluated in FP64
__device__ __forceinline__ bool face_value(float S, float det, float disc, float mv, float am0, float &w, float &s,
                                           float &M) {
    const float p = S * (1.0f / 6.0f);
    const float is = rsqrtf(p);
    s = p * is;
    const float r = 0.5f * det * is * is * is;
    const float om = disc / (S * S * S);                 // 1 - r^2
    w = r > 0.0f ? om / (1.0f + r) : 1.0f - r;
    M = am0 + fabsf(mv) + 2.0f * s;
    const float ms = M * is;
    return om > 4e-8f + 4e-13f * ms * ms * ms && S > 1e-9f;   // S^3 well inside the FP32 range
}

// the least eigenvalues (less m0) of a candidate's two faces, reduced to their
// minimum and the larger bound
__device__ __forceinline__ bool candidate(const df2 (&b)[6], float mv, float am0, float &val, float &err, float &smax) {
    // b: deviators, components 00 01 02 11 12 22 of the (minus, plus) faces
    df2 S = df2_add(df2_mul(b[0], b[0]), df2_mul(b[3], b[3]));
    S = df2_add(S, df2_mul(b[5], b[5]));
    df2 so = df2_add(df2_mul(b[1], b[1]), df2_mul(b[2], b[2]));
    so = df2_add(so, df2_mul(b[4], b[4]));
    S = df2_add(S, scale(so, 2.0f));
    const df2 a0 = df2_sub(df2_mul(b[3], b[5]), df2_mul(b[4], b[4]));
    const df2 a1 = df2_sub(df2_mul(b[1], b[5]), df2_mul(b[4], b[2]));
    const df2 a2 = df2_sub(df2_mul(b[1], b[4]), df2_mul(b[3], b[2]));
    const df2 det = df2_add(df2_sub(df2_mul(b[0], a0), df2_mul(b[1], a1)), df2_mul(b[2], a2));
    // S^3 - 54 det^2 = 216 p^3 (1 - r^2)
    const df2 S3 = df2_mul(df2_mul(S, S), S);
    const df2 d54 = df2_mul(df2_mul(det, det), df2{f2(54.0f), f2(0.0f)});
    const df2 disc = df2_sub(S3, d54);
    float2 w, s, M;
    const bool okx = face_value(S.hi.x, det.hi.x, disc.hi.x, mv, am0, w.x, s.x, M.x);
    const bool oky = face_value(S.hi.y, det.hi.y, disc.hi.y, mv, am0, w.y, s.y, M.y);
    const float2 iu = make_float2(rsqrtf(w.x), rsqrtf(w.y));
    const float2 u = __fmul2_rn(w, iu);
    const float2 lam = __ffma2_rn(s, two_t(u), make_float2(-mv, mv));
    val = fminf(lam.x, lam.y);
    const float amv = fabsf(mv);
    const float rx = M.x / s.x, ry = M.y / s.y;
    const float ex = s.x * (4e-6f + 1e-11f * iu.x) + 1e-6f * amv + 1e-13f * M.x * rx * (1.0f + rx * iu.x);
    const float ey = s.y * (4e-6f + 1e-11f * iu.y) + 1e-6f * amv + 1e-13f * M.y * ry * (1.0f + ry * iu.y);
    err = fmaxf(ex, ey);
    smax = fmaxf(s.x, s.y);
    return okx && oky;
}

// A cell's C, its deviator and mean
struct CellC {
    df c[6], b[6], m;
    float am;
};
__device__ __forceinline__ df third_df() { return df{0.3333333433f, -9.934107758e-09f}; }
__device__ __forceinline__ void cell_split(CellC &c) {
    c.m = df_mul(df_add(df_add(c.c[0], c.c[3]), c.c[5]), third_df());
    c.am = fabsf(c.m.hi);
#pragma unroll
    for (int m = 0; m < 6; ++m) c.b[m] = (m == 0 || m == 3 || m == 5) ? df_sub(c.c[m], c.m) : c.c[m];
}

// The candidate code (0..2, 3 for the cell value) of one direction, or -1 when
// rounding could change the FP64 choice.  dv: the differences (c0 - c-, c+ - c0).
__device__ __forceinline__ int choose(const CellC &c, df2 (&dv)[6]) {
    const df2 mean = df2_mul(df2_add(df2_add(dv[0], dv[3]), dv[5]), dup(third_df()));
    dv[0] = df2_sub(dv[0], mean);
    dv[3] = df2_sub(dv[3], mean);
    dv[5] = df2_sub(dv[5], mean);
    float val[3], err[3], s = 0.0f;
    bool ok = true;
#pragma unroll
    for (int l = 0; l < 3; ++l) {
        // v = (c+ - c0)/2, (c0 - c-)/2, (c+ - c-)/4 for l = 0, 1, 2; the faces
        // are c0 - v and c0 + v
        df2 b[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const df e = l == 0 ? df2_y(dv[m]) : (l == 1 ? df2_x(dv[m]) : df_add(df2_x(dv[m]), df2_y(dv[m])));
            const float w = l == 2 ? 0.25f : 0.5f;
            const float eh = w * e.hi, el = w * e.lo;
            b[m] = df2_add(dup(c.b[m]), df2{make_float2(-eh, eh), make_float2(-el, el)});
        }
        const float mv = l == 0 ? 0.5f * mean.hi.y : (l == 1 ? 0.5f * mean.hi.x : 0.25f * (mean.hi.x + mean.hi.y));
        float sl;
        ok = candidate(b, mv, c.am, val[l], err[l], sl) && ok;
        s = fmaxf(s, sl);
    }
    const int best = val[1] > val[0] ? (val[2] > val[1] ? 2 : 1) : (val[2] > val[0] ? 2 : 0);
    const float vb = best == 0 ? val[0] : (best == 1 ? val[1] : val[2]);
    const float eb = best == 0 ? err[0] : (best == 1 ? err[1] : err[2]);
    bool clear = true;
#pragma unroll
    for (int l = 0; l < 3; ++l) clear = clear && (l == best || vb - val[l] > eb + err[l]);
    const float e0 = fmaxf(err[0], fmaxf(err[1], err[2])) + 2e-7f * (c.am + s), lam = c.m.hi + vb;
    if (ok && lam < -e0) return 3;
    return ok && clear && lam > e0 ? best : -1;
}

}  // namespace codes
}  // namespace f8
