// ks_gradient.cuh -- the rows of the gradient and the adjoint of one step (sample_adjoint, transport.jl:221-245).
#pragma once
#include "ks_transfer.cuh"

namespace ks {

// ---- per-splat constants of the gradient (FP64) ------------------------------------------------
enum GradTab { GT_DF0, GT_DKR, GT_DBT0, GT_DBT1, GT_DBT2, GT_DBP0, GT_DBP1, GT_DBP2, GT_QW, GT_QX, GT_QY, GT_QZ, GT_QN, GT_COUNT };

// gradient rows of a THERMAL21 column (polarized.jl:17-19, 0-based)
enum GradRow { GR_X, GR_Y, GR_Z, GR_S1, GR_S2, GR_S3, GR_Q1, GR_Q2, GR_Q3, GR_Q4, GR_T0, GR_LOGW, GR_LOGNE, GR_LOGTE, GR_LOGB,
               GR_THB, GR_PHB, GR_U1, GR_U2, GR_U3, GR_OMEGA, GR_COUNT };

// ---- the step adjoint (sample_adjoint, transport.jl:221-245) -------------------------------------
// in: j (4), alpha (4), rho (3) of the sample summed over elements, Dl the step length; w the adjoint
// in front of the sample, R the tail behind it. out: O (for w <- O^T w), E = Ej j, and c-bar =
// (j-bar 4, alpha-bar 4, rho-bar 3).
template <class T>
__device__ __forceinline__ void sample_adjoint(const MomentCoeffs& MC, const T* in, T Dl, const T w[4], const T R[4], T O[16], T E[4],
                                               T cb[11]) {
    using D = Dual<T, 7>;
    D al[4], rh[3];
#pragma unroll
    for (int q = 0; q < 4; ++q) al[q] = D::seed(in[4 + q], q);
#pragma unroll
    for (int q = 0; q < 3; ++q) rh[q] = D::seed(in[8 + q], 4 + q);
    D Od[16], Ejd[16];
    step_operator(MC, al, rh, D(Dl), Od, Ejd);
    D qd(T(0));
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        D row = Od[4 * r] * R[0] + Od[4 * r + 1] * R[1] + Od[4 * r + 2] * R[2] + Od[4 * r + 3] * R[3] +
                Ejd[4 * r] * in[0] + Ejd[4 * r + 1] * in[1] + Ejd[4 * r + 2] * in[2] + Ejd[4 * r + 3] * in[3];
        qd += row * w[r];
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) O[q] = Od[q].v;
#pragma unroll
    for (int r = 0; r < 4; ++r) E[r] = Ejd[4 * r].v * in[0] + Ejd[4 * r + 1].v * in[1] + Ejd[4 * r + 2].v * in[2] + Ejd[4 * r + 3].v * in[3];
#pragma unroll
    for (int c = 0; c < 4; ++c) cb[c] = Ejd[c].v * w[0] + Ejd[4 + c].v * w[1] + Ejd[8 + c].v * w[2] + Ejd[12 + c].v * w[3];
#pragma unroll
    for (int q = 0; q < 7; ++q) cb[4 + q] = qd.d[q];
}

// ---- the step adjoint in structured form (the mixed path) -----------------------------------------
// In every branch of the step operator O = sum_n o_n K^n and Ej = s sum_n e_n K^n (n = 0..3), with K
// the rescaled matrix K' of step_operator (without alpha_I) and scalar coefficients that depend on
// alpha, rho only through the invariants a = aI D, a2 = |alpha_QUV|^2, r2 = |rho|^2, ar = alpha.rho
// (step.jl:64-124). So q = w^T (O R + Ej j) has
//   dq/dtheta = sum_n [do_n/dtheta <w, K^n R> + o_n <w, dK^n/dtheta R>] + s (the same with e_n and j),
// the coefficient partials by four duals in (a, a2, r2, ar), and dK/dtheta a constant sparse matrix:
// <w, dK^2 v> = <w, G K v> + <K^T w, G v>, <w, dK^3 v> = <w, G K^2 v> + <K^T w, G K v> + <K^2T w, G v>.

// sample_adjoint (transport.jl:221-245) with the structured partials; same outputs as sample_adjoint
template <class T>
__device__ __forceinline__ void sample_adjoint_structured(const MomentCoeffs& MC, const T* in, T Dl, const T w[4], const T R[4], T O[16],
                                                          T E[4], T cb[11]) {
    const T s = pow2_below(Dl);
    const T D = Dl / s;
    const T aI = in[4] * s, aQ = in[5] * s, aU = in[6] * s, aV = in[7] * s, rQ = in[8] * s, rU = in[9] * s, rV = in[10] * s;
    using D4 = Dual<T, 4>;
    const D4 a = D4::seed(aI * D, 0), a2 = D4::seed(aQ * aQ + aU * aU + aV * aV, 1), r2 = D4::seed(rQ * rQ + rU * rU + rV * rV, 2),
             ar = D4::seed(aQ * rQ + aU * rU + aV * rV, 3);
    D4 o[4], e[4];
    step_coefficients(MC, a, a2, r2, ar, D, o, e);
    T K[16];
    K[0] = 0; K[1] = aQ; K[2] = aU; K[3] = aV; K[4] = aQ; K[5] = 0; K[6] = rV; K[7] = -rU;
    K[8] = aU; K[9] = -rV; K[10] = 0; K[11] = rQ; K[12] = aV; K[13] = rU; K[14] = -rQ; K[15] = 0;
    const T* jv = in;
    T KR[4], K2R[4], K3R[4], Kj[4], K2j[4], K3j[4], Kw[4], K2w[4];
    kmul(K, R, KR); kmul(K, KR, K2R); kmul(K, K2R, K3R);
    kmul(K, jv, Kj); kmul(K, Kj, K2j); kmul(K, K2j, K3j);
    kmul_t(K, w, Kw); kmul_t(K, Kw, K2w);
    const T P[4] = {dot4(w, R), dot4(w, KR), dot4(w, K2R), dot4(w, K3R)};
    const T J[4] = {dot4(w, jv), dot4(w, Kj), dot4(w, K2j), dot4(w, K3j)};
    // the values: O = sum o_n K^n, E = s sum e_n K^n j, j-bar = Ej^T w = s sum e_n (K^n)^T w
    {
        T K2[16];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) K2[4 * i + jj] = K[4 * i] * K[jj] + K[4 * i + 1] * K[4 + jj] + K[4 * i + 2] * K[8 + jj] + K[4 * i + 3] * K[12 + jj];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const T k3 = K2[4 * i] * K[jj] + K2[4 * i + 1] * K[4 + jj] + K2[4 * i + 2] * K[8 + jj] + K2[4 * i + 3] * K[12 + jj];
                O[4 * i + jj] = ((i == jj) ? o[0].v : T(0)) + o[1].v * K[4 * i + jj] + o[2].v * K2[4 * i + jj] + o[3].v * k3;
            }
        T K3w[4];
        kmul_t(K, K2w, K3w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            E[i] = s * (e[0].v * jv[i] + e[1].v * Kj[i] + e[2].v * K2j[i] + e[3].v * K3j[i]);
            cb[i] = s * (e[0].v * w[i] + e[1].v * Kw[i] + e[2].v * K2w[i] + e[3].v * K3w[i]);
        }
    }
    // through the invariants
    T dx[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        T acc = T(0);
#pragma unroll
        for (int n = 0; n < 4; ++n) acc += o[n].d[x] * P[n] + s * e[n].d[x] * J[n];
        dx[x] = acc;
    }
    T g[7];
    g[0] = dx[0] * D;                                   // aI
    g[1] = dx[1] * T(2) * aQ + dx[3] * rQ;              // aQ
    g[2] = dx[1] * T(2) * aU + dx[3] * rU;
    g[3] = dx[1] * T(2) * aV + dx[3] * rV;
    g[4] = dx[2] * T(2) * rQ + dx[3] * aQ;              // rQ
    g[5] = dx[2] * T(2) * rU + dx[3] * aU;
    g[6] = dx[2] * T(2) * rV + dx[3] * aV;
    // through the explicit K of K^1, K^2, K^3
    T f1[6], f2a[6], f2b[6], f3a[6], f3b[6], f3c[6];
    T h1[6], h2a[6], h2b[6], h3a[6], h3b[6], h3c[6];
    kgen_forms(w, R, f1); kgen_forms(w, KR, f2a); kgen_forms(Kw, R, f2b);
    kgen_forms(w, K2R, f3a); kgen_forms(Kw, KR, f3b); kgen_forms(K2w, R, f3c);
    kgen_forms(w, jv, h1); kgen_forms(w, Kj, h2a); kgen_forms(Kw, jv, h2b);
    kgen_forms(w, K2j, h3a); kgen_forms(Kw, Kj, h3b); kgen_forms(K2w, jv, h3c);
#pragma unroll
    for (int t = 0; t < 6; ++t)
        g[1 + t] += o[1].v * f1[t] + o[2].v * (f2a[t] + f2b[t]) + o[3].v * (f3a[t] + f3b[t] + f3c[t]) +
                    s * (e[1].v * h1[t] + e[2].v * (h2a[t] + h2b[t]) + e[3].v * (h3a[t] + h3b[t] + h3c[t]));
    // d/d(alpha_true) = s d/d(alpha_scaled)
#pragma unroll
    for (int t = 0; t < 7; ++t) cb[4 + t] = s * g[t];
}

}  // namespace ks
