// f8_adjoint_mixed.cu — discrete adjoint of the FP32-mixed 3D step (the
// gradient of f8_grad on an F8_MIXED context).
//
// The mixed step (f8_step_mixed.cu) computes the same discrete operator as
// the FP64 step; it differs in precision and in how it reaches the same
// solutions (increment-form Helmholtz solves, a Neumann / Sherman-Morrison
// Newton iteration converging to the same root, an FP32 pressure solve with a
// double-float defect correction).  Its adjoint is therefore the FP64 step's
// stage transposes (f8_adjoint_kernels.cuh), here in FP32 arithmetic on FP32
// adjoint fields, reading the tape the mixed step writes (MixTape): the
// velocity high parts, C before and after the update, the selection codes,
// the explicit IBM velocity, U* and Phi with the boundary values the forward
// kernels read, and the marker forces.  The parameter gradient is accumulated
// in FP64.  The solves are the mixed step's own FP32 transforms and
// tridiagonal sweeps (the operators are symmetric).
#include <algorithm>
#include <cstdio>
#include "f8_adjoint_kernels.cuh"
#include "f8_df64.cuh"
#include "f8_kernels.h"

namespace f8 {

cudaError_t adjoint_fold_state_f(AdjStateF &A, const Dev &d, cudaStream_t s) {
    const Geo &g = d.g;
    return fold_walls(fold_with_c(fold_set<float>({{A.lU, BC_U}, {A.lV, BC_V}, {A.lW, BC_W}, {A.lP, BC_P}}), A.lC, d.cs, 6), g, s);
}

cudaError_t take_interior_f(const float *src, float *dst, const Geo &g, int n, cudaStream_t s) {
    k_take_interior<float><<<(n + 255) / 256, 256, 0, s>>>(src, dst, g, n); count_launch();
    return cudaGetLastError();
}

namespace {

cudaError_t poisson_solve_f(Dev &d, const float *src, float *dst, float *lo, int mode, cudaStream_t s) {
    return d.g.walls ? mixed_solve_walls(d, src, dst, lo, mode, 2, s)
                     : mixed_solve_periodic(d, src, dst, lo, mode, 0.0, -1.0, s);
}

// k_div_adj with the pressure adjoint q as a double-float pair (qh, ql): the
// adjoint projection lU + (q - q(+e))/(d dt) cancels the gradient part of
// lU, so the difference and its scaling are formed in df64 and only the
// result is rounded to FP32
__global__ void k_div_adj_df(const float *__restrict__ lU, const float *__restrict__ lV, const float *__restrict__ lW,
                             const float *__restrict__ qh, const float *__restrict__ ql, DivAdjOut<float> o, Geo g, df cx,
                             df cy, df cz) {
    div_adj_cell<float>(o, g, [&](int h, int xp, int yp, int zp, float &x, float &y, float &z) {
        auto q = [&](int p) { return df{qh[p], ql[p]}; };
        const df q0 = q(h);
        x = df_to_f(df_add_f(df_mul(df_sub(q0, q(xp)), cx), lU[h]));
        y = df_to_f(df_add_f(df_mul(df_sub(q0, q(yp)), cy), lV[h]));
        z = df_to_f(df_add_f(df_mul(df_sub(q0, q(zp)), cz), lW[h]));
    });
}

}  // namespace

cudaError_t step_mixed_adjoint(Dev &d, AdjStateF &A, const MixTape &t, const double *drag_w, bool ab2_first,
                               bool polymer, cudaStream_t s) {
    const Geo &g = d.g;
    const int cs = d.cs;
    const size_t hb = (size_t)cs * sizeof(float);
    const double dt = d.ph.dt, re = d.ph.re, beta = d.ph.beta, wi = d.ph.wi;
    const double kap = dt * beta / re / 2.0;
    dim3 blk(32, 8);
    const AdjCoef<float> kc = adj_coef<float>(g);
    // 6. projection / pressure update
    k_march_adj<float><<<adj_cells(g, blk), blk, 0, s>>>(A.lU, A.lV, A.lW, A.lP, A.pack, t.Phi, g, (float)kap,
                                                         (float)(dt / (2.0 * re)), kc, A.grad); count_launch();
    // 5. Poisson, refined as the forward's pressure solve: q0 = L^-1 r in FP32,
    // the defect r - L_h q0 in df64, q = q0 + L^-1 (defect) as a df64 pair
    F8_CUDA_RET(poisson_solve_f(d, A.pack, A.lQ[0], nullptr, 0, s));
    F8_CUDA_RET(mixed_defect(d, A.lQ[0], A.pack, A.zero, A.rdef, s));
    F8_CUDA_RET(poisson_solve_f(d, A.rdef, A.lQ[0], A.qlo, 2, s));
    DivAdjOut<float> dout{};
    for (int c = 0; c < 3; ++c) { dout.pk[c] = A.pack + (size_t)c * d.ni; dout.lUa[c] = A.lUa[c]; }
    k_div_adj_df<<<adj_cells(g, blk), blk, 0, s>>>(A.lU, A.lV, A.lW, A.lQ[0], A.qlo, dout, g, df_from_d(1.0 / (g.dx * dt)),
                                                   df_from_d(1.0 / (g.dy * dt)), df_from_d(1.0 / (g.dz * dt)));
    count_launch();
    // 4. Helmholtz: the three solves as the forward's parallel branches
    {
        const float *src[3] = {dout.pk[0], dout.pk[1], dout.pk[2]};
        F8_CUDA_RET(mixed_helmholtz(d, 3, src, A.lQ, s));
    }
    // 3. IBM
    if (d.nm > 0) {
        IbmAdjArgs<float> ia{};
        ia.mx = d.mx; ia.my = d.my; ia.mcyl = d.mcyl; ia.nm = d.nm; ia.ncyl = d.ncyl;
        ia.idx = 1.0 / g.dx; ia.idy = 1.0 / g.dy; ia.mvol = d.mvol;
        ia.idvol = 1.0 / ((g.dx * g.dy) * g.dz); ia.dvn = (g.dx * g.dx * g.dx) / ((g.dx * g.dy) * g.dz); ia.cylvol = d.cylvol;
        for (int c = 0; c < 3; ++c) {
            ia.i0[c] = d.mi0[c]; ia.j0[c] = d.mj0[c];
            ia.Ua[c] = t.Ua[c]; ia.Fc[c] = t.Fc[c]; ia.lQ[c] = A.lQ[c]; ia.lUa[c] = A.lUa[c];
        }
        ia.w = drag_w;
        ia.grad = A.grad;
        const IbmAdjShape sh = ibm_adj_shape(d.nm);
        k_ibm_adj<3, float><<<dim3(g.nz, 3, sh.chunks), dim3(32, 3, sh.warps), 0, s>>>(ia, g); count_launch();
    }
    // 2. momentum right-hand side: per-cell sources, then the gather of the
    // velocity, pressure and (with the polymer) C0 / C adjoints
    {
        MomAdjArgs<float> ma{};
        ma.U = t.U; ma.V = t.V; ma.W = t.W;
        for (int c = 0; c < 3; ++c) {
            ma.Up[c] = t.Up[c]; ma.lQ[c] = A.lQ[c]; ma.lUa[c] = A.lUa[c];
            ma.lA0[c] = A.lA0[c]; ma.lT0[c] = A.lT0[c];
        }
        ma.cs = cs; ma.ab2_first = ab2_first ? 1 : 0; ma.polymer = polymer ? 1 : 0;
        ma.vis = (float)(beta / re); ma.coef_t = (float)((1.0 - beta) / (re * wi));
        ma.c_helm = (float)(dt / (2.0 * re)); ma.inv_re = (float)(1.0 / re);
        ma.grad = A.grad;
        ma.kc = kc;
        k_momadj_src<float><<<adj_cells(g, blk), blk, 0, s>>>(ma, A.work, g); count_launch();
        MomGatherArgs<float> mg{};
        mg.U = t.U; mg.V = t.V; mg.W = t.W; mg.src = A.work;
        mg.lU = A.lU; mg.lV = A.lV; mg.lW = A.lW; mg.lP = A.lP; mg.C = t.Cn; mg.lC = A.lC;
        mg.cs = cs; mg.polymer = polymer ? 1 : 0;
        mg.lp2 = (float)(d.ph.lp2); mg.inv_1mb = (float)(1.0 / (1.0 - beta)); mg.inv_wi = (float)(1.0 / wi);
        mg.grad = A.grad;
        mg.kc = kc;
        k_momadj_gather<float><<<adj_rows(g, blk), blk, 0, s>>>(mg, g); count_launch();
    }
    // 1. polymer: per-cell implicit-function adjoint and Cstar weights, then
    // the gather of the adjoint of C^n and of the velocity
    if (polymer) {
        PolyAdjArgs<float> pa{};
        pa.C = t.C; pa.Cn = t.Cn; pa.codes = t.codes; pa.codes_g = t.codes_g; pa.U = t.U; pa.V = t.V; pa.W = t.W;
        pa.lX = A.lC;
        pa.cs = cs; pa.dt = (float)(dt); pa.wi = (float)(wi); pa.lp2 = (float)(d.ph.lp2); pa.grad = A.grad;
        pa.kc = kc; pa.dtwi = (float)(dt / wi); pa.dtwi2 = (float)(dt / (wi * wi));
        const dim3 pb(32, 4);
        k_polyadj_mu<float><<<adj_rows(g, pb), pb, 0, s>>>(pa, A.work, g); count_launch();
        k_polyadj_cstar<float><<<adj_rows(g, blk), blk, 0, s>>>(pa, A.work, g); count_launch();
        PolyGatherArgs<float> pga{};
        pga.src = A.work; pga.lC = A.lC2; pga.lU = A.lU; pga.lV = A.lV; pga.lW = A.lW; pga.cs = cs;
        k_polyadj_gather<float><<<adj_rows(g, blk), blk, 0, s>>>(pga, g); count_launch();
        std::swap(A.lC, A.lC2);
    } else {
        F8_CUDA_RET(cudaMemsetAsync(A.lC, 0, 6 * hb, s));
    }
    return adjoint_fold_state_f(A, d, s);
}

}  // namespace f8
