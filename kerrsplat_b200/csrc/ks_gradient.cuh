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

// In FP32 the partials of the closed forms cancel: they divide differences of cosh b1, cos b2 and the like by
// b1^2 + b2^2, twice: most of the error of a gradient by the pattern rate (64 splats, 224 x 224 x 896: 7.1e-6, and
// 1.2e-6 with the two forms below; the call 22.6 ms with FP32 duals, 20.8 so, 25.8 with FP64 duals for every step that
// is not cubic). The forms:
//   - |K|^2 D^2 <= 1/8 (kSeriesStep): the coefficients are symmetric functions of K's two squared eigenvalues x1, x2 (scaled by D^2),
//     so power series in x1 + x2 = s and x1 x2 = p, four terms (the fifth is below 3e-7 of a partial), without the
//     square root, with exact partials;
//   - stronger steps: FP64 duals, out of line.
// sum_{k>=1} w_k h_{k-1}(x1, x2) -> hi, w_0 - p sum_{k>=2} w_k h_{k-2} -> lo, scaled by ch and cl, with the partials by
// (a2, r2, ar); h_k: complete homogeneous polynomials
template <int N>
__device__ __forceinline__ void series_pair(const float w[5], float s, float p, float ds, float dp, float cl, float ch, Dual<float, N>& lo, Dual<float, N>& hi) {
    const float h2 = s * s - p, h3 = s * (s * s - 2.f * p);
    const float H = w[1] + w[2] * s + w[3] * h2 + w[4] * h3, Hs = w[2] + w[3] * 2.f * s + w[4] * (3.f * s * s - 2.f * p), Hp = -w[3] - 2.f * s * w[4];
    const float G = w[2] + w[3] * s + w[4] * h2, Ls = -p * (w[3] + w[4] * 2.f * s), Lp = p * w[4] - G;
    hi.v = ch * H; hi.d[1] = ch * Hs * ds; hi.d[2] = -hi.d[1]; hi.d[3] = ch * Hp * dp;
    lo.v = cl * (w[0] - p * G); lo.d[1] = cl * Ls * ds; lo.d[2] = -lo.d[1]; lo.d[3] = cl * Lp * dp;
}

static __device__ __noinline__ void step_series(const MomentCoeffs& MC, float a, float a2, float r2, float ar, float D, Dual<float, 4> o[4], Dual<float, 4> e[4]) {
    const float D2 = D * D, ard = ar * D2, s = (a2 - r2) * D2, p = -ard * ard, ds = D2, dp = -2.f * ard * D2, ex = fexp(-a);
    constexpr float c[5] = {1.f, 1.f / 2, 1.f / 24, 1.f / 720, 1.f / 40320}, q[5] = {1.f, 1.f / 6, 1.f / 120, 1.f / 5040, 1.f / 362880};
    float m[11], w[5];
    moment_values(MC, a, ex, m);
    series_pair(c, s, p, ds, dp, ex, ex * D2, o[0], o[2]);
    series_pair(q, s, p, ds, dp, -ex * D, -ex * D * D2, o[1], o[3]);
#pragma unroll
    for (int n = 0; n < 4; ++n) o[n].d[0] = -o[n].v;
    Dual<float, 4> lo, hi;   // by a: M_n -> -M_{n+1}
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = -c[k] * m[2 * k + 1];
    series_pair(w, s, p, ds, dp, D, D * D2, lo, hi);
    e[0].d[0] = lo.v; e[2].d[0] = hi.v;
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = -q[k] * m[2 * k + 2];
    series_pair(w, s, p, ds, dp, -D2, -D2 * D2, lo, hi);
    e[1].d[0] = lo.v; e[3].d[0] = hi.v;
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = c[k] * m[2 * k];
    series_pair(w, s, p, ds, dp, D, D * D2, e[0], e[2]);
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] = q[k] * m[2 * k + 1];
    series_pair(w, s, p, ds, dp, -D2, -D2 * D2, e[1], e[3]);
}

static __device__ __noinline__ void step_wide(const MomentCoeffs& MC, double a, double a2, double r2, double ar, double D, Dual<float, 4> o[4], Dual<float, 4> e[4]) {
    using D4 = Dual<double, 4>;
    D4 od[4], ed[4];
    step_coefficients(MC, D4::seed(a, 0), D4::seed(a2, 1), D4::seed(r2, 2), D4::seed(ar, 3), D, od, ed);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        o[n].v = float(od[n].v); e[n].v = float(ed[n].v);
#pragma unroll
        for (int k = 0; k < 4; ++k) { o[n].d[k] = float(od[n].d[k]); e[n].d[k] = float(ed[n].d[k]); }
    }
}

// sample_adjoint (transport.jl:221-245) with the structured partials; same outputs as sample_adjoint
template <class T>
__device__ __forceinline__ void sample_adjoint_structured(const MomentCoeffs& MC, const T* in, T Dl, const T w[4], const T R[4], T O[16],
                                                          T E[4], T cb[11]) {
    const T s = pow2_below(Dl);
    const T D = Dl / s;
    const T aI = in[4] * s, aQ = in[5] * s, aU = in[6] * s, aV = in[7] * s, rQ = in[8] * s, rU = in[9] * s, rV = in[10] * s;
    using D4 = Dual<T, 4>;
    D4 o[4], e[4];
    if constexpr (is_f32<T>) {
        const T a2 = aQ * aQ + aU * aU + aV * aV, r2 = rQ * rQ + rU * rU + rV * rV;
        if ((a2 + r2) * D * D <= kSeriesStep) step_series(MC, aI * D, a2, r2, aQ * rQ + aU * rU + aV * rV, D, o, e);
        else
            step_wide(MC, double(aI) * D, double(aQ) * aQ + double(aU) * aU + double(aV) * aV, double(rQ) * rQ + double(rU) * rU + double(rV) * rV,
                      double(aQ) * rQ + double(aU) * rU + double(aV) * rV, D, o, e);
    } else {
        step_coefficients(MC, D4::seed(aI * D, 0), D4::seed(aQ * aQ + aU * aU + aV * aV, 1), D4::seed(rQ * rQ + rU * rU + rV * rV, 2),
                          D4::seed(aQ * rQ + aU * rU + aV * rV, 3), D, o, e);
    }
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
