// ks_lib.cu -- libkerrsplat_b200.so: the kernels of the render hot path and the C ABI of
// include/kerrsplat_b200.h.
//
// Pipeline of one context (the device-side GeodesicCache of cache.jl:85-125):
//   ks_regenerate: k_root_case (K0, screen order) -> stable radix sort by root case (4, 2, 0 real
//     roots; cub, deterministic) -> k_build_plan (K1: FP64 per-ray constants, sorted order) ->
//     exclusive scan of anchor counts -> k_anchor_segments (one thread per two anchors of a ray: Jacobi
//     states by the addition theorem, validity, closed-form parts and the Gauss-Legendre integral of the
//     smooth part since the previous anchor) -> k_anchor_prefix (per-ray running sums).
//   ks_thin_image / ks_render: k_splat_table (per-splat FP64 constants) -> k_thin (a block marches 32 rays,
//     in pieces of their depth) or k_stream -> k_transport -> k_compose (ks_transport.cuh) -> k_unsort.
#include <cub/cub.cuh>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/kerrsplat_b200.h"
#include "ks_dft.cuh"
#include "ks_transfer.cuh"

using namespace ks;

static __constant__ MomentCoeffs c_moments;

#include "ks_context.cuh"

namespace {

// ---- kernels: regenerate ---------------------------------------------------------------------------

__global__ void k_root_case(Spacetime st, const double* __restrict__ alpha, const double* __restrict__ beta, long long npix,
                            unsigned char* __restrict__ key, long long* __restrict__ idx) {
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= npix) return;
    RayC R = build_ray(st, alpha[i], beta[i]);
    key[i] = (unsigned char)(4 - R.numreals);   // 4 real roots first (pixel_constants.jl:167-176)
    idx[i] = i;
}

template <class T>
__device__ __forceinline__ MarchRay<T> march_ray_of(const RayCT<T>& R, const SpacetimeT<T>& st, TimeT<T> dtau) {
    MarchRay<T> M;
    M.rcase = R.rcase; M.k = R.k; M.c = R.c; M.fo = R.fo; M.fo_d = R.fo;
    M.m0 = R.map[0]; M.m1 = R.map[1]; M.m2 = R.map[2]; M.m3 = R.map[3];
    M.tau_valid = R.tau_valid; M.dtau = dtau;
    M.pmu = R.pmu; M.pscale = R.pscale; M.tempfac = R.tempfac; M.poffset = R.poffset; M.sqrt_up = R.sqrt_up;
    M.um = R.um; M.up_m_um = R.up_m_um; M.psign = R.psign; M.vortical = R.vortical; M.scattering = R.scattering;
    M.a = st.a; M.lam = R.lam; M.eta = R.eta; M.rp = st.rp; M.rmn = st.rmn; M.sp = R.sp; M.sm = R.sm;
    M.Qt = R.Qt; M.Qtm = R.Qtm; M.Qphi = R.Qphi; M.Qphim = R.Qphim; M.r4 = R.r4; M.qC = R.qC; M.qn = R.qn;
    M.sqrt_eps = R.sqrt_eps; M.gc = R.gc; M.mp = R.mp; M.K2 = R.K2;
    M.vabsalpha = R.vabsalpha; M.valpha2 = R.valpha2; M.vabsbeta = R.vabsbeta; M.vabscos = st.abscos; M.vcos2 = st.cos2;
    M.pa = st.a;
    return M;
}

template <class T>
__device__ __forceinline__ JS<T> xr_at(const RayCT<T>& R, TimeT<T> tau) { return jstate(R.c * (R.fo - tau), R.k); }
template <class T>
__device__ __forceinline__ JS<T> xt_at(const RayCT<T>& R, TimeT<T> tau) { return jstate(R.pscale * (tau + R.poffset) / R.tempfac, R.pmu); }

__global__ void k_build_plan(Spacetime st, const double* __restrict__ alpha, const double* __restrict__ beta,
                             const long long* __restrict__ perm, long long npix, long long npad, double* __restrict__ f,
                             long long* __restrict__ nanch_out) {
    long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    long long i = perm[j];
    RayC R = build_ray(st, alpha[i], beta[i]);
    auto put = [&](int field, double v) { f[field * npad + j] = v; };
    int Nj = st.N;
    if (st.density > 0.0) {
        const double want = 64.0 * ceil(st.density * R.tau_total / 64.0);
        Nj = (want > 0.0) ? int(fmin(double(st.N), fmax(double(st.nmin), want))) : st.nmin;
    }
    double dtau = R.tau_total / (Nj + 1);
    double h = dtau / 2.0;
    int Man = anchor_interval(st.M, 1.0 - R.k);
    int nanch = (Nj - 1) / Man + 1;
    put(PF_NSAMP, Nj);
    put(PF_ALPHA, R.alpha); put(PF_BETA, R.beta); put(PF_ETA, R.eta); put(PF_LAM, R.lam);
    put(PF_NUMREALS, R.numreals); put(PF_CASE, R.rcase);
    put(PF_K, R.k); put(PF_C, R.c); put(PF_FO, R.fo);
    put(PF_MAP0, R.map[0]); put(PF_MAP1, R.map[1]); put(PF_MAP2, R.map[2]); put(PF_MAP3, R.map[3]);
    put(PF_TAU_VALID, R.tau_valid); put(PF_TAU_TOTAL, R.tau_total); put(PF_DTAU, dtau);
    put(PF_PMU, R.pmu); put(PF_PSCALE, R.pscale); put(PF_TEMPFAC, R.tempfac); put(PF_POFFSET, R.poffset);
    put(PF_SQRTUP, R.sqrt_up); put(PF_UM, R.um); put(PF_UPMUM, R.up_m_um); put(PF_PSIGN, R.psign);
    put(PF_VORTICAL, R.vortical ? 1.0 : 0.0); put(PF_GTHO, R.gtho);
    put(PF_SP, R.sp); put(PF_SM, R.sm); put(PF_QT, R.Qt); put(PF_QTM, R.Qtm); put(PF_QPHI, R.Qphi); put(PF_QPHIM, R.Qphim);
    put(PF_R4, R.r4); put(PF_SCATTER, R.scattering ? 1.0 : 0.0);
    put(PF_QC, R.qC); put(PF_QN, R.qn); put(PF_SQRTEPS, R.sqrt_eps); put(PF_GC, R.gc); put(PF_MP, R.mp); put(PF_K2, R.K2);
    put(PF_VABSALPHA, R.vabsalpha); put(PF_VALPHA2, R.valpha2); put(PF_VABSBETA, R.vabsbeta);
    JS<double> dr = jstep_constants(-R.c * h, R.k);
    JS<double> dth = jstep_constants(R.pscale * h / R.tempfac, R.pmu);
    put(PF_DR_SN, dr.sn); put(PF_DR_CN, dr.cn); put(PF_DR_DN, dr.dn);
    put(PF_DTH_SN, dth.sn); put(PF_DTH_CN, dth.cn); put(PF_DTH_DN, dth.dn);
    // the interval that holds the radial turning point of a scattering ray (quadrature.jl:269)
    int turn_k = -1;
    if (R.scattering) {
        for (int k = 2; k <= Nj; ++k) {
            double ta = (k - 1) * dtau, tb = k * dtau;
            if (ta < R.fo && R.fo < tb) { turn_k = k; break; }
        }
    }
    put(PF_TURN_K, turn_k);
    if (turn_k > 0) {
        double ta = (turn_k - 1) * dtau, tb = turn_k * dtau;
        JS<double> a1 = xr_at(R, (ta + R.fo) / 2.0), b1 = xt_at(R, (ta + R.fo) / 2.0);
        JS<double> a2 = xr_at(R, (R.fo + tb) / 2.0), b2 = xt_at(R, (R.fo + tb) / 2.0);
        JS<double> pt = xt_at(R, R.fo);
        put(PF_P1R_SN, a1.sn); put(PF_P1R_CN, a1.cn); put(PF_P1R_DN, a1.dn);
        put(PF_P1T_SN, b1.sn); put(PF_P1T_CN, b1.cn); put(PF_P1T_DN, b1.dn);
        put(PF_P2R_SN, a2.sn); put(PF_P2R_CN, a2.cn); put(PF_P2R_DN, a2.dn);
        put(PF_P2T_SN, b2.sn); put(PF_P2T_CN, b2.cn); put(PF_P2T_DN, b2.dn);
        put(PF_PTT_SN, pt.sn); put(PF_PTT_CN, pt.cn); put(PF_PTT_DN, pt.dn);
    } else {
        for (int q = PF_P1R_SN; q <= PF_PTT_DN; ++q) put(q, 0.0);
    }
    put(PF_MANCHOR, Man); put(PF_NANCH, nanch);
    put(PF_R1RE, R.rre[0]); put(PF_R1IM, R.rim[0]); put(PF_R2RE, R.rre[1]); put(PF_R2IM, R.rim[1]);
    put(PF_R3RE, R.rre[2]); put(PF_R3IM, R.rim[2]); put(PF_R4RE, R.rre[3]); put(PF_R4IM, R.rim[3]);
    nanch_out[j] = nanch;
}

// The smooth integrands at tau from direct Jacobi states, the t part in its large-r form past r = 64.
template <class T>
__device__ __forceinline__ void anchor_integrand(const RayCT<T>& R, const MarchRay<T>& M, TimeT<T> tau, T& gt, T& gp) {
    JS<T> xr = xr_at(R, tau), xt = xt_at(R, tau);
    Point<T> p = ray_point(M, xr, xt, tau);
    gt = p.gt; gp = p.gphi;
    T r = p.r, a = M.a, lam = M.lam;
    T P = r * r + a * a - a * lam;
    if (r > 64.0 && P > 0.0) {
        T D = r * r - 2.0 * r + a * a;
        T Qv = M.eta + (lam - a) * (lam - a);
        T as = fabs(p.s);
        T diff = D * Qv / (P + as) * (1.0 + 2.0 / r) + 2.0 * (2.0 * r - a * a) * P / (r * D);
        T s2 = 1.0 - p.cth * p.cth;
        T wp = p.s * M.rp / (r * (r - M.rp)) / M.sp;
        T wm = p.s * M.rmn / (r * (r - M.rmn)) / M.sm;
        gt = diff + a * (lam - a * s2) - M.Qt * wp - M.Qtm * wm;
    }
}

__constant__ double c_gl_x[16];
__constant__ double c_gl_w[16];

template <class T>
__device__ void gl_panel(const RayCT<T>& R, const MarchRay<T>& M, TimeT<T> ta, TimeT<T> tb, T& It, T& Ip) {
    const TimeT<T> mid = 0.5 * (ta + tb), half = 0.5 * (tb - ta);
    T st = T(0.0), sp = T(0.0);
    for (int i = 0; i < 16; ++i) {
        T gt, gp;
        anchor_integrand(R, M, mid + half * c_gl_x[i], gt, gp);
        st += c_gl_w[i] * gt; sp += c_gl_w[i] * gp;
    }
    It = half * st; Ip = half * sp;
}

constexpr int kAnchorPanelSamples = 4;

// The Landen scale of one modulus: the amplitude of any argument without the scale's square roots again.
struct AmScale {
    double ratio[12], top;
    int n;
    __device__ explicit AmScale(double m) {
        double a = 1.0, b = sqrt(1.0 - m), c = sqrt(m);
        n = 0;
        while (n < 11 && c > kEps * a) {
            const double a1 = 0.5 * (a + b);
            c = c * c / (4.0 * a1);
            b = sqrt(a * b);
            a = a1;
            ratio[n++] = c / a;
        }
        top = ldexp(a, n);
    }
    __device__ JS<double> state(double u, double mu) const {
        double ph = top * u;
        for (int i = n - 1; i >= 0; --i) ph = 0.5 * (ph + asin(ratio[i] * sin(ph)));
        double s, c;
        sincos(ph, &s, &c);
        return {s, c, sqrt(fma(-mu, s * s, 1.0))};
    }
};

// jstep with one reciprocal
__device__ __forceinline__ JS<double> jadd(const JS<double>& x, const JS<double>& d, double mu) {
    const double inv = 1.0 / (1.0 - mu * (x.sn * x.sn) * (d.sn * d.sn));
    return {(x.sn * d.cn * d.dn + d.sn * x.cn * x.dn) * inv, (x.cn * d.cn - x.sn * x.dn * d.sn * d.dn) * inv,
            (x.dn * d.dn - mu * x.sn * x.cn * d.sn * d.cn) * inv};
}

// The per-ray factors of the smooth integrands (smooth() in their FP64 form) and the integrands at a pair
// of Jacobi states: the horizon factors share one reciprocal, Delta = (r - r_+)(r - r_-), and cos theta
// enters through its square only.
struct AnchorRates {
    double wpf, wmf, Q, qp, qpm, poln, ips;
    __device__ AnchorRates(const MarchRay<double>& M)
        : wpf(M.rp / M.sp), wmf(M.rmn / M.sm), Q(M.eta + (M.lam - M.a) * (M.lam - M.a)), qp(M.Qphi), qpm(M.Qphim), poln(M.lam * M.qC),
          ips(1.0 / M.pscale) {}
    __device__ void at(const MarchRay<double>& M, const JS<double>& xr, const JS<double>& xt, bool inbound, double& gt, double& gp) const {
        const double a = M.a, lam = M.lam, r = radius(M, xr);
        const double di = 1.0 / xt.dn, sn = xt.sn * di * ips, cn = xt.cn * di, sn2 = sn * sn;
        const double c2 = fmin(1.0, M.vortical ? fmax(M.um + M.up_m_um * sn2, 0.0) : M.sqrt_up * M.sqrt_up * sn2);
        const double dp = r - M.rp, dm = r - M.rmn, D = dp * dm, P = r * r + a * a - a * lam;
        const double as = sqrt(fmax(P * P - D * Q, 0.0)), s = inbound ? -as : as;
        const double i = 1.0 / (r * D);
        const double wp = s * wpf * dm * i, wm = s * wmf * dp * i;
        double t;
        if (r > 64.0 && P > 0.0) t = D * Q / (P + as) * (1.0 + 2.0 * D * i) + 2.0 * (2.0 * r - a * a) * P * i;
        else t = (r * r + a * a) * P * (r * i) - as * (1.0 + 2.0 * D * i);
        gt = t + a * (lam - a * (1.0 - c2)) - M.Qt * wp - M.Qtm * wm;
        gp = a * (2.0 * r - a * lam) * (r * i) - qp * wp - qpm * wm + poln * (1.0 - M.gc * di * (1.0 - 0.5 * M.mp * cn * cn)) / (1.0 - M.qn * sn2);
    }
};

// The anchors of a ray, kAnchorRun consecutive ones a thread (the whole warp at the same place of
// neighbouring rays). A panel's sixteen Gauss-Legendre states come from its middle's by the addition
// theorem, with steps that all panels of the ray share, and the middle of the next panel from this one's;
// only the panel that holds the radial turning point (cut in two there) and the first of all, up to the
// first sample, evaluate amplitudes at their own nodes. Bound by FP64 arithmetic: an amplitude costs some
// seven sines and arcsines, and the kernel that took two per node spent 32.1 ms at 65536 rays x 1024 samples.
constexpr int kAnchorRun = 2;

__global__ void __launch_bounds__(kBlock) k_anchor_segments(PlanView P, Spacetime st, long long npix, double* __restrict__ anchors) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    const int nanch = int(P.get(PF_NANCH, j));
    const int m0 = blockIdx.y * kAnchorRun, m1 = min(nanch, m0 + kAnchorRun);
    if (m0 >= nanch) return;
    const MarchRay<double> M = load_ray<double>(P, st, j);
    const AnchorRates rates(M);
    const AmScale sr(M.k), sq(M.pmu);
    const int Man = M.Manchor;
    const double dtau = M.dtau, fo = M.fo_d;
    const double kr = M.c, kt = M.pscale / M.tempfac;   // arguments: c (fo - tau) and pscale (tau + offset) / tempfac
    auto xr_at_ = [&](double tau) { return sr.state(kr * (fo - tau), M.k); };
    auto xt_at_ = [&](double tau) { return sq.state(kt * (tau + M.poffset), M.pmu); };
    // a panel by amplitudes at its own nodes
    auto panel = [&](double ta, double tb, double& It, double& Ip) {
        const double mid = 0.5 * (ta + tb), half = 0.5 * (tb - ta);
        double s0 = 0.0, s1 = 0.0;
        for (int i = 0; i < 16; ++i) {
            const double tau = mid + half * c_gl_x[i];
            double gt, gp;
            rates.at(M, xr_at_(tau), xt_at_(tau), tau < fo, gt, gp);
            s0 += c_gl_w[i] * gt; s1 += c_gl_w[i] * gp;
        }
        It += half * s0; Ip += half * s1;
    };
    const JS<double> x0 = xt_at_(0.0);
    const double pc0 = polar_closed(M, 0.0, x0.sn / (M.pscale * x0.dn), x0.cn / x0.dn);
    // the shared steps: the nodes' distances from the middle of a panel (symmetric about it), panel to panel
    const int np = (Man + kAnchorPanelSamples - 1) / kAnchorPanelSamples;
    const double hp = Man * dtau / np, half = 0.5 * hp;
    JS<double> nr[8], nt[8], pr, pt;
    if (m1 > 1) {
        for (int i = 0; i < 8; ++i) {
            const double d = half * fabs(c_gl_x[i]);
            nr[i] = sr.state(kr * d, M.k); nt[i] = sq.state(kt * d, M.pmu);
        }
        pr = sr.state(-kr * hp, M.k); pt = sq.state(kt * hp, M.pmu);
    }
    for (int m = m0; m < m1; ++m) {
        const int k = 1 + m * Man;
        const double tau = k * dtau;
        double* A = anchors + (M.anchor_off + m) * AF_COUNT;
        const JS<double> xr = xr_at_(tau), xt = xt_at_(tau);
        A[AF_XR_SN] = xr.sn; A[AF_XR_CN] = xr.cn; A[AF_XR_DN] = xr.dn;
        A[AF_XT_SN] = xt.sn; A[AF_XT_CN] = xt.cn; A[AF_XT_DN] = xt.dn;
        double th, cth; bool nu;
        polar_cos(M, xt, th, cth, nu);
        const bool reached = tau <= M.tau_valid;
        A[AF_OK] = (reached && visible(M, cth)) ? 1.0 : 0.0;
        A[AF_PAD] = 0.0;
        double lead_t = 0.0, lead_p = 0.0, It = 0.0, Ip = 0.0;
        if (reached) {
            // closed-form parts at tau, accumulated from the observer
            const double r = radius(M, xr);
            const double F = r + 2.0 * log(r);
            const double L = (M.scattering && tau > fo) ? F - 2.0 * (M.r4 + 2.0 * log(M.r4)) : -F;
            const double lp = log((r - st.rp) / r) / M.sp, lm = log((r - st.rmn) / r) / M.sm;
            lead_t = L + M.Qt * lp + M.Qtm * lm;
            lead_p = M.Qphi * lp + M.Qphim * lm + polar_closed(M, tau, xt.sn / (M.pscale * xt.dn), xt.cn / xt.dn) - pc0;
            // smooth part over (previous anchor, tau]
            if (m == 0) {
                panel(0.0, (M.scattering && fo < tau) ? fo : tau, It, Ip);
                if (M.scattering && fo < tau) panel(fo, tau, It, Ip);
            } else {
                const double ta = (1 + (m - 1) * Man) * dtau;
                JS<double> yr = xr_at_(ta + half), yt = xt_at_(ta + half);
                int split = -1;
                for (int q = 0; q < np; ++q) {
                    if (q > 0) { yr = jadd(yr, pr, M.k); yt = jadd(yt, pt, M.pmu); }
                    const double a0 = ta + q * hp, mid = a0 + half;
                    if (M.scattering && a0 < fo && fo < a0 + hp) { split = q; continue; }   // after the loop: the warp stays together
                    const bool inbound = mid < fo;
                    double s0 = 0.0, s1 = 0.0;
#pragma unroll 1
                    for (int i = 0; i < 8; ++i) {
                        // tau = mid -+ d: the radial argument runs backwards
                        const JS<double> dr = nr[i], dt = nt[i], er = {-dr.sn, dr.cn, dr.dn}, et = {-dt.sn, dt.cn, dt.dn};
                        double g0, p0, g1, p1;
                        rates.at(M, jadd(yr, dr, M.k), jadd(yt, et, M.pmu), inbound, g0, p0);
                        rates.at(M, jadd(yr, er, M.k), jadd(yt, dt, M.pmu), inbound, g1, p1);
                        s0 += c_gl_w[i] * (g0 + g1); s1 += c_gl_w[i] * (p0 + p1);
                    }
                    It += half * s0; Ip += half * s1;
                }
                if (split >= 0) {
                    panel(ta + split * hp, fo, It, Ip);
                    panel(fo, split == np - 1 ? tau : ta + (split + 1) * hp, It, Ip);
                }
            }
        }
        A[AF_T] = lead_t; A[AF_PHI] = lead_p;
        A[AF_SEG_T] = It; A[AF_SEG_PHI] = Ip;
    }
}

__global__ void k_anchor_prefix(long long npix, long long npad, const double* __restrict__ f, const long long* __restrict__ aoff,
                                double* __restrict__ anchors) {
    long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    int nanch = int(f[PF_NANCH * npad + j]);
    double st = 0.0, sp = 0.0;
    for (int m = 0; m < nanch; ++m) {
        double* A = anchors + (aoff[j] + m) * AF_COUNT;
        st += A[AF_SEG_T]; sp += A[AF_SEG_PHI];
        A[AF_T] += st; A[AF_PHI] += sp;
    }
}

// ---- kernels: splat tables ---------------------------------------------------------------------------

// K0 and K1 from K_nu(x) = int_0^inf exp(-x cosh t) cosh(nu t) dt by the trapezoidal rule.
__host__ __device__ void besselk01(double x, double& k0, double& k1) {
    // trapezoid in t on exp(-x (cosh t - 1)) (the factor exp(-x) applied at the end); the step
    // resolves the Gaussian core of width 1/sqrt(x) (error ~ exp(-2 pi^2 / (x h^2)) < 1e-17)
    const double h = fmin(0.125, 0.6 / sqrt(x));
    double s0 = 0.5, s1 = 0.5;
    for (int j = 1; j < 20000; ++j) {
        double t = j * h;
        double ch = cosh(t);
        double e = exp(-x * (ch - 1.0));
        s0 += e;
        s1 += e * ch;
        if (e < 1e-18 * s0) break;
    }
    double ex = exp(-x);
    k0 = h * s0 * ex; k1 = h * s1 * ex;
}

struct SetDesc {
    int kind, nrows, nsplat, first;   // first = index of its first splat in the concatenated table
    const double* params;
    const double* hyp;
    double gmax;
    int koff, nk;                     // knot splats: offset of the set's first knot record, knot count
    const double* knots;              // the knot array (device)
};

__global__ void k_splat_table(SetDesc d, double* __restrict__ tab) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nsplat) return;
    const double* p = d.params + (long long)d.nrows * i;
    double* o = tab + (long long)(d.first + i) * ST_COUNT;
    for (int q = 0; q < ST_COUNT; ++q) o[q] = 0.0;
    o[ST_KIND] = d.kind;
    o[ST_CX] = p[0]; o[ST_CY] = p[1]; o[ST_CZ] = p[2];
    o[ST_T0] = p[10]; o[ST_OMEGA] = p[d.nrows - 1];
    o[ST_ES1] = exp(-p[3]); o[ST_ES2] = exp(-p[4]); o[ST_ES3] = exp(-p[5]);
    double q1 = p[6], q2 = p[7], q3 = p[8], q4 = p[9];
    double n = sqrt(q1 * q1 + q2 * q2 + q3 * q3 + q4 * q4);
    double w = q1 / n, x = q2 / n, y = q3 / n, z = q4 / n;
    o[ST_R0] = 1 - 2 * (y * y + z * z); o[ST_R1] = 2 * (x * y - w * z); o[ST_R2] = 2 * (x * z + w * y);
    o[ST_R3] = 2 * (x * y + w * z); o[ST_R4] = 1 - 2 * (x * x + z * z); o[ST_R5] = 2 * (y * z - w * x);
    o[ST_R6] = 2 * (x * z - w * y); o[ST_R7] = 2 * (y * z + w * x); o[ST_R8] = 1 - 2 * (x * x + y * y);
    o[ST_INVW] = exp(-p[11]);
    double smax = fmax(p[3], fmax(p[4], p[5]));
    o[ST_SUPP] = (-2.0 * log(kWEIGHT_CUTOFF)) * exp(2 * smax);
    o[ST_RHO] = sqrt(p[0] * p[0] + p[1] * p[1]);
    o[ST_KOFF] = d.kind == KS_KNOT21 ? double(d.koff + 4 * d.nk * i) : 0.0;
    o[ST_NK] = d.kind == KS_KNOT21 ? double(d.nk) : 0.0;
    if (d.kind == KS_KNOT21) {
        // every interpolated centre lies in the box of the knots: a point farther than the box's
        // half-diagonal plus the support radius from its centre is outside the support at any time
        const double* kn = d.knots + d.koff + 4 * d.nk * i;
        double lo[3], hi[3], half2 = 0.0;
        for (int q = 0; q < 3; ++q) {
            lo[q] = hi[q] = kn[(q + 1) * d.nk];
            for (int k = 1; k < d.nk; ++k) { lo[q] = fmin(lo[q], kn[(q + 1) * d.nk + k]); hi[q] = fmax(hi[q], kn[(q + 1) * d.nk + k]); }
            half2 += 0.25 * (hi[q] - lo[q]) * (hi[q] - lo[q]);
        }
        o[ST_CX] = 0.5 * (lo[0] + hi[0]); o[ST_CY] = 0.5 * (lo[1] + hi[1]); o[ST_CZ] = 0.5 * (lo[2] + hi[2]);
        const double rb = sqrt(half2) + sqrt(o[ST_SUPP]);
        o[ST_RHO] = rb * rb;   // the bounding radius squared (knot splats use no pattern circle)
    }
    if (d.kind == KS_THIN14) { o[ST_LOGA] = p[12]; return; }
    o[ST_NE] = exp(p[12]);
    double Bmag, thB, phB, u1, u2, u3;
    if (d.kind == KS_THERMAL21 || d.kind == KS_KNOT21) {
        double Te = exp(p[13]);
        o[ST_TE] = Te;
        double k0, k1;
        besselk01(1.0 / Te, k0, k1);
        double xb = 1.0 / Te;
        double k2 = k0 + 2.0 * k1 / xb;
        o[ST_F0] = k2 > 0 ? k0 / k2 : 1.0;
        o[ST_KR] = k2 > 0 ? k1 / k2 : 1.0;
        Bmag = exp(p[14]); thB = p[15]; phB = p[16]; u1 = p[17]; u2 = p[18]; u3 = p[19];
    } else {
        Bmag = exp(p[15]); thB = p[16]; phB = p[17]; u1 = p[18]; u2 = p[19]; u3 = p[20];
        if (d.kind == KS_POWERLAW22) {
            double pp = p[13], gmin = exp(p[14]);
            o[ST_P] = pp; o[ST_GMIN] = gmin; o[ST_GMAX] = d.gmax;
            o[ST_GSPAN] = pow(gmin, 1 - pp) - pow(d.gmax, 1 - pp);
            o[ST_GAMJ] = tgamma((3 * pp - 1) / 12) * tgamma((3 * pp + 19) / 12);
            o[ST_GAMA] = tgamma((3 * pp + 2) / 12) * tgamma((3 * pp + 22) / 12);
        } else {
            double kap = p[13], wk = exp(p[14]);
            o[ST_KAP] = kap; o[ST_W] = wk; o[ST_HYP] = d.hyp ? d.hyp[i] : 0.0;
            o[ST_G43] = tgamma(kap - 4.0 / 3); o[ST_G2] = tgamma(kap - 2);
            o[ST_GQ] = tgamma(kap / 4 - 1.0 / 3); o[ST_GP] = tgamma(kap / 4 + 4.0 / 3);
            o[ST_GK2] = tgamma(2 + kap / 2);
            double k0, k1;
            besselk01(1.0 / wk, k0, k1);
            double xb = 1.0 / wk;
            double k2 = k0 + 2.0 * k1 / xb;
            o[ST_KB] = k0 / (k2 + 1e-40);
        }
    }
    double B[3] = {Bmag * sin(thB) * cos(phB), Bmag * sin(thB) * sin(phB), Bmag * cos(thB)};
    double Bn = sqrt(B[0] * B[0] + B[1] * B[1] + B[2] * B[2]);
    o[ST_BMAG] = Bmag;
    if (Bn > 0) { o[ST_BHX] = B[0] / Bn; o[ST_BHY] = B[1] / Bn; o[ST_BHZ] = B[2] / Bn; o[ST_BZERO] = 0.0; }
    else { o[ST_BHX] = 0; o[ST_BHY] = 0; o[ST_BHZ] = 1; o[ST_BZERO] = 1.0; }
    o[ST_U1] = u1; o[ST_U2] = u2; o[ST_U3] = u3;
}

// ---- kernels: the fused march with its consumers -----------------------------------------------------

}  // namespace

namespace {

struct StoreSink {
    double *t, *r, *th, *ph; unsigned char* fl;
    long long npix, j;
    __device__ void operator()(int k, const Sample<double>& s) {
        long long q = (long long)(k - 1) * npix + j;
        t[q] = s.t; r[q] = s.r; th[q] = s.theta; ph[q] = s.phi;
        fl[q] = (s.ok ? 1 : 0) | (s.nur ? 2 : 0) | (s.nutheta ? 4 : 0);
    }
};

__global__ void k_march_store(PlanView P, Spacetime st, long long npix, double* t, double* r, double* th, double* ph,
                              unsigned char* fl, double* resid_t, double* resid_phi) {
    long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    MarchRay<double> R = load_ray<double>(P, st, j);
    StoreSink sink{t, r, th, ph, fl, npix, j};
    double rt, rp;
    march(P, st, j, R, sink, rt, rp);
    resid_t[j] = rt; resid_phi[j] = rp;
}

// ThinRenderer (Splats.jl:113-128) over rows of kThinRow values: the centre, t0, omega, 1 / w, ln A, and the whitened
// rotation R diag(exp(-s)) formed in FP64.
constexpr int kThinRow = 16;
template <class T>
__device__ __forceinline__ T thin_row(const double* p, int f) {
    constexpr int head[7] = {ST_CX, ST_CY, ST_CZ, ST_T0, ST_OMEGA, ST_INVW, ST_LOGA};
    return f < 7 ? T(p[head[f]]) : T(p[ST_R0 + f - 7] * p[ST_ES1 + (f - 7) % 3]);
}

template <class T>
struct ThinSink {
    const T* rows; int nsplat; T t_obs; T a, rh_lo; T dtau; T acc;
    T eta, lam;
    __device__ void operator()(int, const Sample<T>& s) {
        if (!(s.ok && rh_lo < s.r && s.r < T(1e3))) return;
        // sin theta from cos theta: the march's angle would be one acos, sin and cos more per sample
        const T cth = s.cos_theta, sth = sqrt(fmax((T(1) - cth) * (T(1) + cth), T(0)));
        T x, y, z;
        ks_position(a, s.r, sth, cth, s.phi, x, y, z);
        const T t = t_obs - s.t;
        T jt = T(0);
        for (int i = 0; i < nsplat; ++i) {
            const T* p = rows + i * kThinRow;
            const T dt = t - p[3];
            T sp, cp;
            fsincos(p[4] * dt, sp, cp);
            const T d0 = x - (p[0] * cp - p[1] * sp), d1 = y - (p[0] * sp + p[1] * cp), d2 = z - p[2];
            const T b0 = d0 * cp + d1 * sp, b1 = -d0 * sp + d1 * cp;
            const T e0 = p[7] * b0 + p[10] * b1 + p[13] * d2, e1 = p[8] * b0 + p[11] * b1 + p[14] * d2, e2 = p[9] * b0 + p[12] * b1 + p[15] * d2;
            const T tt = dt * p[5];
            jt += exp(p[6] - (e0 * e0 + e1 * e1 + e2 * e2 + tt * tt) / T(2));
        }
        SampleFrame<T> F = sample_frame(a, s.r, T(0), sth, cth, eta, lam, s.nur, s.nutheta);
        T g = T(1) / F.pz[0];
        T Sg = s.r * s.r + a * a * cth * cth;
        acc += g * g * jt * Sg * dtau;
    }
};

// The thin image: a block marches 32 rays (march_block), each thread taking a quarter of their samples, over one of
// nseg pieces of their depth. One piece writes the image; with more, each leaves its sums (and anchor residuals) in
// `part` [3][nseg][npix] for k_thin_sum. Bound by FP64 arithmetic on a full screen (every sample rotates every splat's
// centre and exponentiates) and by the latency of the march on a small one. Whole calls, one thread a ray against these
// blocks: 24 x 24 rays x 64 samples x 3 splats 560 : 260 us, 128 x 128 x 512 x 12 splats 6.09 : 2.49 ms.
template <class T>
__global__ void __launch_bounds__(kBlock, sizeof(T) == 4 ? 4 : 3)
k_thin(PlanView P, Spacetime st, long long npix, const double* __restrict__ tab64, int nsplat, double t_obs, int nseg, double* __restrict__ part,
       const long long* __restrict__ perm, double* __restrict__ out, double* __restrict__ resid_t, double* __restrict__ resid_phi) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[kMarchWarps][32];
    MarchShared<T>& shared = *reinterpret_cast<MarchShared<T>*>(smem);
    T* rows = reinterpret_cast<T*>(smem + (sizeof(MarchShared<T>) + 15) / 16 * 16);
    for (int q = threadIdx.x; q < nsplat * kThinRow; q += kBlock) rows[q] = thin_row<T>(tab64 + (q / kThinRow) * ST_COUNT, q % kThinRow);
    const int lane = threadIdx.x & 31, seg = blockIdx.y;
    const bool live = blockIdx.x * 32LL + lane < npix;
    const long long j = live ? blockIdx.x * 32LL + lane : npix - 1;
    const int nsamp = int(P.get(PF_NSAMP, j));
    // pieces of whole re-anchoring intervals: each starts from the anchor table
    const int len = ((nsamp + nseg - 1) / nseg + st.M - 1) / st.M * st.M;
    ThinSink<T> sink{rows, nsplat, T(t_obs), T(st.a), T(st.rh * (1 + 1e-3)), T(P.get(PF_DTAU, j)), T(0), T(P.get(PF_ETA, j)), T(P.get(PF_LAM, j))};
    double rt, rp;
    march_block<true>(P, st, j, live, 1 + seg * len, 1 + (seg + 1) * len, shared, sink, rt, rp);   // its first barrier is behind the rows
    red[threadIdx.x >> 5][lane] = double(sink.acc);
    __syncthreads();
    if (threadIdx.x >= 32 || !live) return;
    double acc = 0.0;
    for (int w = 0; w < kMarchWarps; ++w) acc += red[w][lane];
    if (nseg > 1) {
        part[seg * npix + j] = acc; part[(nseg + seg) * npix + j] = rt; part[(2 * nseg + seg) * npix + j] = rp;
        return;
    }
    out[perm ? perm[j] : j] = acc;   // sorted order, or screen order through the permutation
    if (resid_t) { resid_t[j] = rt; resid_phi[j] = rp; }
}

__global__ void k_thin_sum(long long npix, int nseg, const double* __restrict__ part, const long long* __restrict__ perm, double* __restrict__ out,
                           double* __restrict__ resid_t, double* __restrict__ resid_phi) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    double acc = 0.0, rt = 0.0, rp = 0.0;
    for (int s = 0; s < nseg; ++s) {
        acc += part[s * npix + j];
        rt = fmax(rt, part[(nseg + s) * npix + j]);
        rp = fmax(rp, part[(2 * nseg + s) * npix + j]);
    }
    out[perm ? perm[j] : j] = acc;
    if (resid_t) { resid_t[j] = rt; resid_phi[j] = rp; }
}

// Pieces of a screen's depth: until there are four blocks per SM, down to one re-anchoring interval each (up to 16).
int thin_pieces(const Spacetime& st, long long npix, int nsm) {
    int nseg = 1;
    while (nseg < 16 && (npix + 31) / 32 * nseg < 4 * nsm && 2 * nseg * (long long)st.M <= st.N) nseg *= 2;
    return nseg;
}

// The allocation-free thin-image variant (ks_thin_image_noalloc) keeps its splat table in this
// file-scope device array instead of a context buffer and runs k_thin with the image written straight
// into the caller's buffer. Every GPU that loads the library holds the array until the process exits;
// every call overwrites the first nsplat rows before reading them; calls that overlap on the GPU (two
// streams, two host threads) share it and race.
constexpr int kNoAllocMaxSplats = 256;
static __device__ __align__(256) double g_noalloc_tab[kNoAllocMaxSplats * ST_COUNT];

// ---- ipole's RIAF as a fluid model of the polarized consumer ------------------------------------
// The reference's test/riaf_model.jl: a thick disk with power-law density and temperature, a
// toroidal field of equipartition-like strength, Keplerian rotation outside the ISCO and the plunge
// with the ISCO's conserved energy and angular momentum inside it, thermal synchrotron (Pandya
// emissivities when `pandya`, ipole's emission_type 1). One element, evaluated at every sample.
struct RiafModel { double nth0, Te0, disk_h, pow_nth, pow_T, Ne_unit, Te_unit, eps, r_isco, rout; int pandya; };

constexpr double kMP = 1.67262171e-24, kKBOL = 1.3806505e-16;   // constants.jl:3-12

// The coefficients and the local frame of the RIAF at the BL point (r, theta) of a sample, for the
// photon of the sample's frame F; false where the model is empty (r <= r_h + 0.1 or r >= rout).
template <class T>
__device__ __forceinline__ bool riaf_element(const RiafModel& m, T a, T r, T th, T sth, T cth, const SampleFrame<T>& F, T alpha, T beta,
                                             T a_sin_tho, T nu, Coef<T>& cf, LFrame<T>& lf) {
    const T rh = T(1) + sqrt(T(1) - a * a);
    if (!(r > rh + T(0.1) && r < T(m.rout))) return false;
    // density, temperature, field strength (ipole's get_model_ne / thetae / b)
    const T zc = r * cth, rc = r * sth;
    const T hh = T(m.disk_h);
    const T n = T(m.nth0) * exp(-zc * zc / T(2) / rc / rc / hh / hh) * pow(r, T(m.pow_nth)) * T(m.Ne_unit);
    const T Te = T(m.Te0) * pow(r, T(m.pow_T)) * T(m.Te_unit) * T(kKBOL) / (T(kME) * T(kCL) * T(kCL));
    T bmag = sqrt(T(8) * kpi<T>() * T(m.eps) * n * T(kMP) * T(kCL) * T(kCL) / T(6) / r);
    if (bmag == T(0)) bmag = T(1e-6);
    // the Boyer-Lindquist metric at (r, theta) and at (r_isco, theta)
    const T s2 = sth * sth;
    auto gdd = [&](T rr, T& gtt, T& gtp, T& grr, T& gpp) {
        const T S = rr * rr + a * a * cth * cth, D = rr * rr - T(2) * rr + a * a;
        gtt = -(T(1) - T(2) * rr / S); gtp = -T(2) * a * rr * s2 / S; grr = S / D;
        gpp = (rr * rr + a * a + T(2) * a * a * rr * s2 / S) * s2;
    };
    T gtt, gtp, grr, gpp;
    gdd(r, gtt, gtp, grr, gpp);
    T om, ur;
    const T risco = T(m.r_isco);
    if (r < risco) {
        // the plunge: the ISCO's conserved e, l (ipole get_model_fourv)
        T itt, itp, irr, ipp;
        gdd(risco, itt, itp, irr, ipp);
        const T wis = T(1) / (pow(risco, T(1.5)) + a);
        const T nrm = sqrt(-(itt + T(2) * wis * itp + wis * wis * ipp));
        const T u0 = T(1) / nrm, u3 = wis / nrm;
        const T e = itt * u0 + itp * u3, l = itp * u0 + ipp * u3;
        // the inverse metric at (r, theta)
        const T S = r * r + a * a * cth * cth, D = r * r - T(2) * r + a * a;
        const T A = (r * r + a * a) * (r * r + a * a) - a * a * D * s2;
        const T utt = -A / (S * D), utp = -T(2) * a * r / (S * D), urr = D / S, upp = (D - a * a * s2) / (S * D * s2);
        const T Kcon = utt * e * e + T(2) * utp * e * l + upp * l * l;
        const T q = -(T(1) + Kcon) / urr;
        const T urk = -(q > T(0) ? sqrt(q) : T(0));
        const T c0 = utt * e + utp * l, c3 = utp * e + upp * l;
        om = c3 / c0;
        ur = urr * urk;
    } else {
        om = T(1) / (pow(r, T(1.5)) + a);
        ur = T(0);
    }
    const T K = gtt + T(2) * om * gtp + om * om * gpp;
    const T q2 = -(T(1) + ur * ur * grr) / K;
    const T ut = q2 > T(0) ? sqrt(q2) : T(0);
    const T u[4] = {ut, ur, T(0), om * ut};
    // toroidal field projected orthogonal to u, normalised to bmag
    const T BdotU = gtp * u[0] + gpp * u[3];
    T b[4] = {BdotU * u[0], BdotU * u[1], T(0), T(1) + BdotU * u[3]};
    const T bb = gtt * b[0] * b[0] + T(2) * gtp * b[0] * b[3] + grr * b[1] * b[1] + gpp * b[3] * b[3];
    const T bs = bmag / sqrt(bb);
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] *= bs;
    // ZAMO components (t, r, phi, -theta): lapse, sqrt(S/D), varpi (. - omega_frame t), -sqrt(S)
    const T S = r * r + a * a * cth * cth, D = r * r - T(2) * r + a * a;
    const T A = (r * r + a * a) * (r * r + a * a) - a * a * D * s2;
    const T lapse = sqrt(S * D / A), omf = T(2) * a * r / A, varpi = sqrt(A / S) * sth, sSD = sqrt(S / D);
    const T u1 = sSD * u[1], u2 = varpi * (u[3] - omf * u[0]), u3 = T(0);
    const T bz0 = lapse * b[0], bz1 = sSD * b[1], bz2 = varpi * (b[3] - omf * b[0]), bz3 = T(0);
    // the field in the fluid frame: boost_zamo_to_fluid(u) (frames.jl:31-41)
    const T gam = sqrt(T(1) + u1 * u1 + u2 * u2 + u3 * u3), qf = T(1) / (gam + T(1));
    const T ub = u1 * bz1 + u2 * bz2 + u3 * bz3;
    const T f1 = -u1 * bz0 + bz1 + u1 * ub * qf, f2 = -u2 * bz0 + bz2 + u2 * ub * qf, f3 = -u3 * bz0 + bz3 + u3 * ub * qf;
    const T fn = sqrt(f1 * f1 + f2 * f2 + f3 * f3);
    const bool bzero = !(fn > T(0));
    lf = local_frame(F, u1, u2, u3, bzero ? T(0) : f1 / fn, bzero ? T(0) : f2 / fn, bzero ? T(1) : f3 / fn, bzero, alpha, beta, a_sin_tho);
    const T nuf = nu / lf.g;
    T sb, cb;
    if constexpr (is_f32<T>) {
        pitch_sc(lf.cosB, sb, cb);
    } else {
        const T thb = acos(fmin(T(1), fmax(T(-1), lf.cosB)));
        sb = sin(thb); cb = cos(thb);
    }
    // Bessel ratios at 1/Theta_e (K2 = K0 + 2 K1 / x), FP64
    double k0, k1;
    const double xb = 1.0 / double(Te);
    besselk01(xb, k0, k1);
    const double k2 = k0 + 2.0 * k1 / xb;
    const T f0 = k2 > 0 ? T(k0 / k2) : T(1), kr = k2 > 0 ? T(k1 / k2) : T(1);
    cf = thermal_cs(n, Te, f0, kr, bmag, nuf, sb, cb);
    if (m.pandya && sb > T(0)) {
        T jI, jQ, jV;
        pandya_emissivities(n, Te, bmag, nuf, sb, cb, jI, jQ, jV);
        const T Bn = planck(nuf, Te);
        const T invB = Bn > T(0) ? T(1) / Bn : T(0);
        cf.jI = jI; cf.jQ = jQ; cf.jV = jV; cf.aI = jI * invB; cf.aQ = jQ * invB; cf.aV = jV * invB;
    }
    return true;
}

// RadiativeTransport of the RIAF at one frequency (stokes_image, test/test_polarized.jl:54-61): the
// FP64 march, the element and the step in T.
template <class T>
struct RiafSink {
    RiafModel m;
    T nu, Lnu;
    T a, rh_lo, dtau, alpha, beta, eta, lam, a_sin_tho;
    T P[16], S[4];
    unsigned int ev[7];

    __device__ void init() {
        for (int q = 0; q < 16; ++q) P[q] = (q % 5 == 0) ? T(1) : T(0);
        for (int q = 0; q < 4; ++q) S[q] = T(0);
        for (int q = 0; q < 7; ++q) ev[q] = 0;
    }

    __device__ void operator()(int, const Sample<double>& s) {
        ev[0]++;
        if (!(s.ok && T(s.r) > rh_lo)) return;
        ev[1]++;
        const T r = T(s.r), th = T(s.theta);
        const T sth = sin(th), cth = cos(th);
        const SampleFrame<T> F = sample_frame(a, r, th, sth, cth, eta, lam, s.nur, s.nutheta);
        Coef<T> cf;
        LFrame<T> lf;
        ev[2]++;
        if (!riaf_element(m, a, r, th, sth, cth, F, alpha, beta, a_sin_tho, nu, cf, lf)) return;
        ev[3]++; ev[4]++; ev[5]++;
        // screen_coefficients (transport.jl:265-270): cap, invariants at nu/g, rotate by 2 chi
        if (!(cf.jI > T(0) || cf.aI > T(0) || cf.rQ != T(0) || cf.rV != T(0))) return;
        const T fe = cap_factor(cf.jI, cf.jQ, cf.jV, T(0.99));
        const T fa = cap_factor(cf.aI, cf.aQ, cf.aV, T(0.99));
        const T nh = nu / lf.g / T(kNU0);
        const T i2 = T(1) / (nh * nh);
        const T jQ = cf.jQ * fe * i2, aQ = cf.aQ * fa * nh, rQ = cf.rQ * nh;
        const T j4[4] = {cf.jI * i2, jQ * lf.c2c, jQ * lf.s2c, cf.jV * fe * i2};
        const T a4[4] = {nh * cf.aI, aQ * lf.c2c, aQ * lf.s2c, cf.aV * fa * nh};
        const T r3[3] = {rQ * lf.c2c, rQ * lf.s2c, nh * cf.rV};
        const T Dl = Lnu * (r * r + a * a * cth * cth) * dtau;
        ev[6]++;
        T O[16], E[4];
        transfer_step(c_moments, j4, a4, r3, Dl, O, E);
        T Pn[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            S[i] += P[4 * i] * E[0] + P[4 * i + 1] * E[1] + P[4 * i + 2] * E[2] + P[4 * i + 3] * E[3];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                Pn[4 * i + q] = P[4 * i] * O[q] + P[4 * i + 1] * O[4 + q] + P[4 * i + 2] * O[8 + q] + P[4 * i + 3] * O[12 + q];
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) P[q] = Pn[q];
    }
};

// One thread per ray, one frequency per grid row: out[(f npix + j) 4 + stokes] in sorted order.
template <class T>
__global__ void __launch_bounds__(kBlock) k_riaf(PlanView P, Spacetime st, long long npix, RiafModel m, const double* __restrict__ nus,
                                                 double L, double* __restrict__ out, unsigned long long* __restrict__ counters) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    const int f = blockIdx.y;
    MarchRay<double> R = load_ray<double>(P, st, j);
    RiafSink<T> sink;
    sink.m = m;
    const double nh = nus[f] / kNU0;
    sink.nu = T(nus[f]); sink.Lnu = T(L / nh);
    sink.a = T(st.a); sink.rh_lo = T(st.rh * (1 + 1e-3)); sink.dtau = T(R.dtau);
    sink.alpha = T(P.get(PF_ALPHA, j)); sink.beta = T(P.get(PF_BETA, j)); sink.eta = T(R.eta); sink.lam = T(R.lam);
    sink.a_sin_tho = T(st.a * sin(st.thetao));
    sink.init();
    double rt, rp;
    march(P, st, j, R, sink, rt, rp);
    double* o = out + ((long long)f * npix + j) * 4;
    const double n3 = nh * nh * nh;
    o[0] = double(sink.S[0]) * n3; o[1] = double(sink.S[1]) * n3; o[2] = double(sink.S[2]) * n3; o[3] = double(sink.S[3]) * n3;
    if (counters) {
        atomicAdd(&counters[0], (unsigned long long)sink.ev[0]);
        for (int q = 1; q < 7; ++q) atomicAdd(&counters[q], (unsigned long long)sink.ev[q]);
    }
}

}  // namespace

#include "ks_adjoint.cuh"
#include "ks_spacetime.cuh"

namespace {

__global__ void k_inverse_perm(const long long* __restrict__ perm, long long npix, long long* __restrict__ inv) {
    long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j < npix) inv[perm[j]] = j;
}

// sorted slot -> output order, for `nvec` blocks of npix rows of `width` doubles
__global__ void k_unsort(const double* __restrict__ src, const long long* __restrict__ perm, long long npix, int width, int nvec,
                         int to_screen, double* __restrict__ dst) {
    long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    long long total = npix * nvec;
    if (q >= total) return;
    long long v = q / npix, j = q % npix;
    long long dj = to_screen ? perm[j] : j;
    for (int w = 0; w < width; ++w) dst[(v * npix + dj) * width + w] = src[(v * npix + j) * width + w];
}

}  // namespace

// ---- the context ----------------------------------------------------------------------------------------

namespace {

void init_constants() {
    MomentCoeffs mc;
    for (int n = 0; n < 11; ++n) {
        double fact = 1.0;
        for (int m = 0; m < 24; ++m) {
            if (m > 0) fact *= m;
            mc.c[n][m] = ((m % 2) ? -1.0 : 1.0) / (fact * (n + m + 1));
            mc.cf[n][m] = float(mc.c[n][m]);
        }
    }
    cudaMemcpyToSymbol(c_moments, &mc, sizeof mc);
    forward_init(mc);
    reverse_init(mc);
    // 16-point Gauss-Legendre nodes on [-1, 1] (Newton on P_16)
    double x[16], w[16];
    const int n = 16;
    for (int i = 0; i < n; ++i) {
        double z = std::cos(kPi * (i + 0.75) / (n + 0.5)), dp = 0.0;
        for (int it = 0; it < 100; ++it) {
            double p1 = 1.0, p2 = 0.0;
            for (int jj = 1; jj <= n; ++jj) { double p3 = p2; p2 = p1; p1 = ((2.0 * jj - 1.0) * z * p2 - (jj - 1.0) * p3) / jj; }
            dp = n * (z * p1 - p2) / (z * z - 1.0);
            double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-17) break;
        }
        double p1 = 1.0, p2 = 0.0;
        for (int jj = 1; jj <= n; ++jj) { double p3 = p2; p2 = p1; p1 = ((2.0 * jj - 1.0) * z * p2 - (jj - 1.0) * p3) / jj; }
        dp = n * (z * p1 - p2) / (z * z - 1.0);
        x[i] = z; w[i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
    cudaMemcpyToSymbol(c_gl_x, x, sizeof x);
    cudaMemcpyToSymbol(c_gl_w, w, sizeof w);
}

int nrows_of(int kind) {
    switch (kind) {
        case KS_THIN14: return 14;
        case KS_THERMAL21: case KS_KNOT21: return 21;
        case KS_POWERLAW22: case KS_KAPPA22: return 22;
        default: return -1;
    }
}

// The concatenated splat table of a scene (and, with `grad`, the gradient table of its THERMAL21
// splats): validates the sets, stages each set's parameters and runs k_splat_table / k_grad_table.
int build_tables(ks_context* c, const ks_splat_set* sets, int nsets, int* ntot_out, bool grad) {
    int ntot = 0;
    for (int s = 0; s < nsets; ++s) {
        int nr = nrows_of(sets[s].kind);
        if (nr < 0 || sets[s].kind == KS_THIN14) return fail(c, KS_ERR_ARGUMENT, "set %d: unsupported kind %d", s, sets[s].kind);
        if (grad && sets[s].kind != KS_THERMAL21)
            return fail(c, KS_ERR_ARGUMENT, "set %d: the adjoint covers thermal polarized splats (KS_THERMAL21) only", s);
        if (sets[s].nsplat < 0 || (sets[s].nsplat > 0 && !sets[s].params)) return fail(c, KS_ERR_ARGUMENT, "set %d: bad parameters", s);
        if (sets[s].kind == KS_KAPPA22 && sets[s].nsplat > 0 && !sets[s].hyp) return fail(c, KS_ERR_ARGUMENT, "set %d: kappa sets need hyp", s);
        ntot += sets[s].nsplat;
    }
    // the knot array of the knot sets (trajectories.jl:80-111): per splat its times, x, y, z
    std::vector<double> kv;
    std::vector<int> koff(nsets, 0);
    for (int s = 0; s < nsets; ++s) {
        const ks_splat_set& S = sets[s];
        if (S.kind != KS_KNOT21 || S.nsplat == 0) continue;
        if (!S.knots || !S.knot_times || S.nknots < 1) return fail(c, KS_ERR_ARGUMENT, "set %d: knot splats need knots and knot times", s);
        const int nk = S.nknots;
        std::vector<double> ht(nk), hk(size_t(3) * nk * S.nsplat);
        KS_CUDA(c, cudaMemcpy(ht.data(), S.knot_times, ht.size() * sizeof(double), cudaMemcpyDefault));
        KS_CUDA(c, cudaMemcpy(hk.data(), S.knots, hk.size() * sizeof(double), cudaMemcpyDefault));
        for (int k = 0; k < nk; ++k)
            if (!std::isfinite(ht[k]) || (k > 0 && !(ht[k] > ht[k - 1]))) return fail(c, KS_ERR_ARGUMENT, "set %d: knot times must increase", s);
        for (double v : hk) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "set %d: non-finite knot", s);
        koff[s] = int(kv.size());
        for (int i = 0; i < S.nsplat; ++i) {
            kv.insert(kv.end(), ht.begin(), ht.end());
            for (int d = 0; d < 3; ++d)
                for (int k = 0; k < nk; ++k) kv.push_back(hk[d + 3 * (k + size_t(nk) * i)]);
        }
    }
    c->nkv = int(kv.size());
    KS_CUDA(c, c->tab.ensure((size_t(std::max(ntot, 1)) * ST_COUNT + kv.size()) * sizeof(double)));
    if (!kv.empty())
        KS_CUDA(c, cudaMemcpyAsync(c->tab.as<double>() + size_t(ntot) * ST_COUNT, kv.data(), kv.size() * sizeof(double),
                                   cudaMemcpyHostToDevice, c->stream));
    if (grad) KS_CUDA(c, c->gtab.ensure(size_t(std::max(ntot, 1)) * GT_COUNT * sizeof(double)));
    int first = 0;
    for (int s = 0; s < nsets; ++s) {
        const ks_splat_set& S = sets[s];
        if (S.nsplat == 0) continue;
        const int nr = nrows_of(S.kind);
        const void* dh = nullptr;
        // each set is staged into its own device buffer
        std::vector<double> hp(size_t(nr) * S.nsplat);
        KS_CUDA(c, cudaMemcpy(hp.data(), S.params, hp.size() * sizeof(double), cudaMemcpyDefault));
        for (double v : hp) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "set %d: non-finite parameter", s);
        DevBuf tmp;
        KS_CUDA(c, tmp.ensure(hp.size() * sizeof(double) + size_t(S.nsplat) * sizeof(double)));
        KS_CUDA(c, cudaMemcpyAsync(tmp.p, hp.data(), hp.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
        if (S.kind == KS_KAPPA22) {
            double* hd = tmp.as<double>() + hp.size();
            KS_CUDA(c, cudaMemcpyAsync(hd, S.hyp, S.nsplat * sizeof(double), cudaMemcpyDefault, c->stream));
            dh = hd;
        }
        SetDesc d{S.kind, nr, S.nsplat, first, tmp.as<const double>(), (const double*)dh, S.gamma_max > 0 ? S.gamma_max : 1e5, koff[s],
                  S.kind == KS_KNOT21 ? S.nknots : 0, c->tab.as<const double>() + size_t(ntot) * ST_COUNT};
        k_splat_table<<<nblocks(S.nsplat, 64), 64, 0, c->stream>>>(d, c->tab.as<double>());
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
        if (grad) {
            k_grad_table<<<nblocks(S.nsplat, 64), 64, 0, c->stream>>>(S.nsplat, first, tmp.as<const double>(), c->gtab.as<double>());
            c->launches++;
            KS_CUDA(c, cudaGetLastError());
        }
        KS_CUDA(c, cudaStreamSynchronize(c->stream));
        tmp.release();
        first += S.nsplat;
    }
    *ntot_out = ntot;
    return KS_OK;
}

// A kernel's bounded wait that gave up (the device flag, cleared): KS_ERR_TIMEOUT. Bit 1: the
// table-staging copy of a transport or reverse kernel (either precision); bit 2: a wait of the tcgen05 GEMM.
int check_device_flag(ks_context* c, const char* what) {
    unsigned f = 0;
    KS_CUDA(c, cudaMemcpy(&f, c->errflag.p, sizeof(unsigned), cudaMemcpyDeviceToHost));
    if (f) {
        KS_CUDA(c, cudaMemset(c->errflag.p, 0, sizeof(unsigned)));
        return fail(c, KS_ERR_TIMEOUT, "%s: %s", what,
                    (f & 2u) ? "a wait of the tensor-core GEMM gave up" : "a shared-memory staging copy did not complete");
    }
    return KS_OK;
}

// The thin image from the splat table `tab` into `out` (through `perm` if given); `resid`: with the anchor residuals.
// Allocates nothing: the pieces' sums have their place since regenerate.
template <class T>
int launch_thin(ks_context* c, const double* tab, int nsplat, double t_obs, const long long* perm, double* out, bool resid) {
    const int nseg = thin_pieces(c->st, c->npix, c->nsm);
    const size_t smem = (sizeof(MarchShared<T>) + 15) / 16 * 16 + size_t(nsplat) * kThinRow * sizeof(T);
    double* rt = resid ? c->resid_t.as<double>() : nullptr;
    double* rp = resid ? c->resid_phi.as<double>() : nullptr;
    KS_CUDA(c, cudaFuncSetAttribute(k_thin<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    k_thin<T><<<dim3(nblocks(c->npix, 32), nseg), kBlock, smem, c->stream>>>(plan_view(c), c->st, c->npix, tab, nsplat, t_obs, nseg,
                                                                            c->thin_part.as<double>(), perm, out, rt, rp);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    if (nseg > 1) {
        k_thin_sum<<<nblocks(c->npix), kBlock, 0, c->stream>>>(c->npix, nseg, c->thin_part.as<double>(), perm, out, rt, rp);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    return KS_OK;
}

// Write `nvec` x npix x width doubles from the sorted device buffer to `out` (host or device) in `order`.
int emit(ks_context* c, const double* sorted, int width, int nvec, int order, double* out) {
    size_t bytes = size_t(c->npix) * width * nvec * sizeof(double);
    bool dev = is_device_ptr(out);
    double* dst = out;
    if (!dev) { KS_CUDA(c, c->stage_out.ensure(bytes)); dst = c->stage_out.as<double>(); }
    long long total = c->npix * nvec;
    k_unsort<<<nblocks(total), kBlock, 0, c->stream>>>(sorted, c->perm.as<long long>(), c->npix, width, nvec,
                                                       order == KS_ORDER_SCREEN ? 1 : 0, dst);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    if (!dev) KS_CUDA(c, cudaMemcpyAsync(out, dst, bytes, cudaMemcpyDeviceToHost, c->stream));
    return KS_OK;
}

}  // namespace

// ---- C ABI -------------------------------------------------------------------------------------------

extern "C" {

int ks_context_create(int device, int flags, ks_context** out) {
    (void)flags;
    if (!out) return KS_ERR_ARGUMENT;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) { cudaGetLastError(); return KS_ERR_DEVICE; }
    if (cudaSetDevice(device) != cudaSuccess) return KS_ERR_DEVICE;
    ks_context* c = new ks_context();
    c->device = device;
    if (cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) { delete c; return KS_ERR_DEVICE; }
    if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) { delete c; return KS_ERR_DEVICE; }
    cudaEventCreate(&c->ev0);
    cudaEventCreate(&c->ev1);
    cudaEventCreate(&c->evc0);
    cudaEventCreate(&c->evc1);
    cudaEventCreate(&c->evg0);
    cudaEventCreate(&c->evg1);
    if (c->errflag.ensure(sizeof(unsigned)) != cudaSuccess || cudaMemset(c->errflag.p, 0, sizeof(unsigned)) != cudaSuccess) {
        delete c;
        return KS_ERR_DEVICE;
    }
    init_constants();
    if (cudaGetLastError() != cudaSuccess) { delete c; return KS_ERR_DEVICE; }
    *out = c;
    return KS_OK;
}

int ks_context_destroy(ks_context* c) {
    if (!c) return KS_OK;
    cudaSetDevice(c->device);
    for (DevBuf* b : {&c->alpha, &c->beta, &c->key, &c->key2, &c->idx, &c->perm, &c->plan, &c->nanch, &c->aoff, &c->anchors,
                      &c->resid_t, &c->resid_phi, &c->scratch, &c->tab, &c->combos, &c->out_sorted, &c->stage_in, &c->stage_out, &c->counters, &c->seg_out, &c->work, &c->stream_buf, &c->inv_perm, &c->dft_tu, &c->dft_tv,
                      &c->dft_a, &c->dft_t, &c->dft_c, &c->dft_s, &c->dft_partial})
        b->release();
    for (DevBuf& b : c->dft_in) b.release();
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->evc0) cudaEventDestroy(c->evc0);
    if (c->evc1) cudaEventDestroy(c->evc1);
    if (c->evg0) cudaEventDestroy(c->evg0);
    if (c->evg1) cudaEventDestroy(c->evg1);
    if (c->ev1) cudaEventDestroy(c->ev1);
    for (cudaGraphExec_t g : {c->graph_exec, c->cgraph_exec})
        if (g) cudaGraphExecDestroy(g);
    for (cudaGraph_t g : {c->graph, c->cgraph})
        if (g) cudaGraphDestroy(g);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return KS_OK;
}

const char* ks_last_error(const ks_context* c) { return c ? c->err.c_str() : "null context"; }

int ks_context_stream(ks_context* c, void** stream) {
    if (!c || !stream) return KS_ERR_ARGUMENT;
    *stream = (void*)c->stream;
    return KS_OK;
}

// Accumulated device time of the render kernels (k_thin / k_transport) since the last reset, and
// the number of launches of this library's kernels.
int ks_kernel_stats(ks_context* c, double* render_ms, long long* render_launches, long long* all_launches, int reset) {
    if (!c) return KS_ERR_ARGUMENT;
    if (render_ms) *render_ms = c->kernel_ms;
    if (render_launches) *render_launches = c->kernel_launches;
    if (all_launches) *all_launches = c->launches;
    if (reset) { c->kernel_ms = 0.0; c->kernel_launches = 0; c->launches = 0; }
    return KS_OK;
}

// Test hook of the staging error path: while on, the transport and reverse kernels arm their table-staging barrier
// without issuing the copy, so the bounded wait runs out and the call fails with KS_ERR_TIMEOUT.
int ks_set_stage_test(ks_context* c, int32_t on) {
    if (!c) return KS_ERR_ARGUMENT;
    c->stage_test = on ? 1 : 0;
    return KS_OK;
}

int ks_gemm_stats(ks_context* c, double* ms, long long* launches, double* flops, int reset) {
    if (!c) return KS_ERR_ARGUMENT;
    if (ms) *ms = c->gemm_ms;
    if (launches) *launches = c->gemm_launches;
    if (flops) *flops = c->gemm_flops;
    if (reset) { c->gemm_ms = 0.0; c->gemm_launches = 0; c->gemm_flops = 0.0; }
    return KS_OK;
}

int ks_set_tensor_path(ks_context* c, int32_t path) {
    if (!c) return KS_ERR_ARGUMENT;
    if (path != KS_TENSOR_TCGEN05 && path != KS_TENSOR_MMA_SYNC) return fail(c, KS_ERR_ARGUMENT, "unknown tensor path %d", path);
    c->tensor_path = path;
    return KS_OK;
}

// Device time of k_transport alone in the mixed ks_render calls since the last reset, and its launches.
int ks_consume_stats(ks_context* c, double* consume_ms, long long* launches, int reset) {
    if (!c) return KS_ERR_ARGUMENT;
    if (consume_ms) *consume_ms = c->consume_ms;
    if (launches) *launches = c->consume_launches;
    if (reset) { c->consume_ms = 0.0; c->consume_launches = 0; }
    return KS_OK;
}

// Count the work events of the following ks_render calls (samples, valid samples, splat tests,
// weights, coefficient evaluations, frames, steps) into a device counter; ks_event_counts reads them.
int ks_set_event_counting(ks_context* c, int on) {
    if (!c) return KS_ERR_ARGUMENT;
    c->count_events = on != 0;
    return KS_OK;
}

int ks_event_counts(ks_context* c, unsigned long long out[7]) {
    if (!c || !out) return KS_ERR_ARGUMENT;
    if (!c->counters.p) { for (int q = 0; q < 7; ++q) out[q] = 0; return KS_OK; }
    KS_CUDA(c, cudaMemcpy(out, c->counters.p, 7 * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    return KS_OK;
}

int ks_camera_set(ks_context* c, const double* alpha, const double* beta, int64_t npix, int32_t nalpha, int32_t nbeta) {
    if (!c) return KS_ERR_ARGUMENT;
    if (!alpha || !beta || npix <= 0) return fail(c, KS_ERR_ARGUMENT, "camera needs at least one pixel");
    if ((long long)nalpha * nbeta != npix) return fail(c, KS_ERR_ARGUMENT, "camera pixel vectors do not match the screen size");
    KS_CUDA(c, cudaSetDevice(c->device));
    std::vector<double> ha(npix), hb(npix);
    KS_CUDA(c, cudaMemcpy(ha.data(), alpha, npix * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(hb.data(), beta, npix * sizeof(double), cudaMemcpyDefault));
    for (long long i = 0; i < npix; ++i)
        if (!std::isfinite(ha[i]) || !std::isfinite(hb[i])) return fail(c, KS_ERR_NONFINITE, "non-finite screen coordinate at pixel %lld", i);
    c->npix = npix;
    c->npad = (npix + 31) / 32 * 32;
    c->nalpha = nalpha; c->nbeta = nbeta;
    KS_CUDA(c, c->alpha.ensure(npix * sizeof(double)));
    KS_CUDA(c, c->beta.ensure(npix * sizeof(double)));
    KS_CUDA(c, cudaMemcpy(c->alpha.p, ha.data(), npix * sizeof(double), cudaMemcpyHostToDevice));
    KS_CUDA(c, cudaMemcpy(c->beta.p, hb.data(), npix * sizeof(double), cudaMemcpyHostToDevice));
    c->regenerated = false;
    return KS_OK;
}

namespace {
int regenerate_impl(ks_context* c, double a, double theta_o, int32_t nsamples, int32_t anchor_M, double density, int32_t nmin);
}

int ks_regenerate(ks_context* c, double a, double theta_o, int32_t nsamples, int32_t anchor_M) {
    return regenerate_impl(c, a, theta_o, nsamples, anchor_M, 0.0, 0);
}

int ks_regenerate_uneven(ks_context* c, double a, double theta_o, double samples_per_mino, int32_t nmin, int32_t nmax, int32_t anchor_M) {
    if (!c) return KS_ERR_ARGUMENT;
    if (!(std::isfinite(samples_per_mino) && samples_per_mino > 0)) return fail(c, KS_ERR_ARGUMENT, "samples per unit Mino time must be positive");
    if (nmin < 1 || nmax < nmin) return fail(c, KS_ERR_ARGUMENT, "need 1 <= nmin <= nmax");
    return regenerate_impl(c, a, theta_o, nmax, anchor_M, samples_per_mino, nmin);
}

int ks_get_nsamples(ks_context* c, int32_t* out) {
    if (!c || !out) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    std::vector<double> f(c->npix);
    KS_CUDA(c, cudaMemcpy(f.data(), c->plan.as<double>() + size_t(PF_NSAMP) * c->npad, c->npix * sizeof(double), cudaMemcpyDeviceToHost));
    std::vector<int32_t> o(c->npix);
    for (long long j = 0; j < c->npix; ++j) o[j] = int32_t(f[j]);
    KS_CUDA(c, cudaMemcpy(out, o.data(), o.size() * sizeof(int32_t), cudaMemcpyDefault));
    return KS_OK;
}

}  // extern "C"

namespace {
int regenerate_impl(ks_context* c, double a, double theta_o, int32_t nsamples, int32_t anchor_M, double density, int32_t nmin) {
    if (!c) return KS_ERR_ARGUMENT;
    if (c->npix <= 0) return fail(c, KS_ERR_ARGUMENT, "set a camera before regenerate");
    ks_graph_destroy(c);   // a captured render holds the old geometry's launch shape
    if (!std::isfinite(a) || !std::isfinite(theta_o)) return fail(c, KS_ERR_NONFINITE, "non-finite spin or inclination");
    if (!(a > 0.0 && a < 1.0)) return fail(c, KS_ERR_ARGUMENT, "spin must lie in (0, 1) (the analytic polar solution divides by a)");
    if (nsamples < 1) return fail(c, KS_ERR_ARGUMENT, "need at least one sample per ray");
    if (anchor_M < 1) return fail(c, KS_ERR_ARGUMENT, "re-anchoring interval must be positive");
    KS_CUDA(c, cudaSetDevice(c->device));
    const long long n = c->npix, npad = c->npad;
    Spacetime& st = c->st;
    st.a = a; st.thetao = theta_o;
    st.rp = 1.0 + std::sqrt(1.0 - a * a); st.rmn = 1.0 - std::sqrt(1.0 - a * a); st.rh = st.rp;
    st.abscos = std::fabs(std::cos(theta_o)); st.cos2 = std::cos(theta_o) * std::cos(theta_o);
    st.N = nsamples; st.M = anchor_M;
    st.density = density; st.nmin = nmin;
    KS_CUDA(c, c->key.ensure(n)); KS_CUDA(c, c->key2.ensure(n));
    KS_CUDA(c, c->idx.ensure(n * sizeof(long long))); KS_CUDA(c, c->perm.ensure(n * sizeof(long long)));
    k_root_case<<<nblocks(n), kBlock, 0, c->stream>>>(st, c->alpha.as<double>(), c->beta.as<double>(), n, c->key.as<unsigned char>(),
                                                        c->idx.as<long long>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    size_t tmp = 0;
    KS_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, tmp, c->key.as<unsigned char>(), c->key2.as<unsigned char>(),
                                               c->idx.as<long long>(), c->perm.as<long long>(), (int)n, 0, 3, c->stream));
    KS_CUDA(c, c->scratch.ensure(tmp));
    KS_CUDA(c, cub::DeviceRadixSort::SortPairs(c->scratch.p, tmp, c->key.as<unsigned char>(), c->key2.as<unsigned char>(),
                                               c->idx.as<long long>(), c->perm.as<long long>(), (int)n, 0, 3, c->stream));
    KS_CUDA(c, c->plan.ensure(size_t(PF_COUNT) * npad * sizeof(double)));
    KS_CUDA(c, c->nanch.ensure(n * sizeof(long long)));
    KS_CUDA(c, c->aoff.ensure((n + 1) * sizeof(long long)));
    k_build_plan<<<nblocks(n), kBlock, 0, c->stream>>>(st, c->alpha.as<double>(), c->beta.as<double>(), c->perm.as<long long>(), n, npad,
                                                         c->plan.as<double>(), c->nanch.as<long long>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    tmp = 0;
    KS_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tmp, c->nanch.as<long long>(), c->aoff.as<long long>(), (int)n, c->stream));
    KS_CUDA(c, c->scratch.ensure(tmp));
    KS_CUDA(c, cub::DeviceScan::ExclusiveSum(c->scratch.p, tmp, c->nanch.as<long long>(), c->aoff.as<long long>(), (int)n, c->stream));
    // totals and case ranges
    std::vector<long long> hn(n), ho(n);
    std::vector<unsigned char> hk(n);
    KS_CUDA(c, cudaMemcpyAsync(hn.data(), c->nanch.p, n * sizeof(long long), cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(ho.data(), c->aoff.p, n * sizeof(long long), cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(hk.data(), c->key2.p, n, cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    c->total_anchors = ho[n - 1] + hn[n - 1];
    c->max_nanch = 0;
    for (long long j = 0; j < n; ++j) c->max_nanch = std::max<int>(c->max_nanch, (int)hn[j]);
    long long cnt[3] = {0, 0, 0};
    for (long long j = 0; j < n; ++j) cnt[hk[j] / 2]++;
    c->ranges[0] = 0; c->ranges[1] = cnt[0];
    c->ranges[2] = cnt[0]; c->ranges[3] = cnt[0] + cnt[1];
    c->ranges[4] = cnt[0] + cnt[1]; c->ranges[5] = n;
    KS_CUDA(c, c->anchors.ensure(size_t(c->total_anchors) * AF_COUNT * sizeof(double)));
    dim3 grid(nblocks(n), (c->max_nanch + kAnchorRun - 1) / kAnchorRun);
    k_anchor_segments<<<grid, kBlock, 0, c->stream>>>(plan_view(c), st, n, c->anchors.as<double>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    k_anchor_prefix<<<nblocks(n), kBlock, 0, c->stream>>>(n, npad, c->plan.as<double>(), c->aoff.as<long long>(), c->anchors.as<double>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    KS_CUDA(c, c->inv_perm.ensure(n * sizeof(long long)));
    k_inverse_perm<<<nblocks(n), kBlock, 0, c->stream>>>(c->perm.as<long long>(), n, c->inv_perm.as<long long>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    KS_CUDA(c, c->resid_t.ensure(n * sizeof(double)));
    if (const int pieces = thin_pieces(st, n, c->nsm); pieces > 1) KS_CUDA(c, c->thin_part.ensure(3 * size_t(pieces) * n * sizeof(double)));
    KS_CUDA(c, c->resid_phi.ensure(n * sizeof(double)));
    KS_CUDA(c, cudaMemsetAsync(c->resid_t.p, 0, n * sizeof(double), c->stream));
    KS_CUDA(c, cudaMemsetAsync(c->resid_phi.p, 0, n * sizeof(double), c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    c->regenerated = true;
    return KS_OK;
}
}  // namespace

extern "C" {

int ks_get_perm(ks_context* c, int64_t* perm) {
    if (!c || !perm) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    KS_CUDA(c, cudaMemcpy(perm, c->perm.p, c->npix * sizeof(long long), cudaMemcpyDefault));
    return KS_OK;
}

int ks_get_ranges(ks_context* c, int64_t ranges[6]) {
    if (!c || !ranges) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    for (int q = 0; q < 6; ++q) ranges[q] = c->ranges[q];
    return KS_OK;
}

int ks_get_residuals(ks_context* c, double* rt, double* rp) {
    if (!c || !rt || !rp) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    KS_CUDA(c, cudaMemcpy(rt, c->resid_t.p, c->npix * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(rp, c->resid_phi.p, c->npix * sizeof(double), cudaMemcpyDefault));
    return KS_OK;
}

int ks_get_ray_constants(ks_context* c, double* out) {
    if (!c || !out) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    const long long n = c->npix, np = c->npad;
    std::vector<double> f(size_t(PF_COUNT) * np);
    KS_CUDA(c, cudaMemcpy(f.data(), c->plan.p, f.size() * sizeof(double), cudaMemcpyDeviceToHost));
    std::vector<double> o(size_t(n) * 24);
    const int fields[24] = {PF_ETA, PF_LAM, PF_NUMREALS, PF_K, PF_C, PF_FO, PF_TAU_TOTAL, PF_TAU_VALID, PF_GTHO,
                            PF_R1RE, PF_R1IM, PF_R2RE, PF_R2IM, PF_R3RE, PF_R3IM, PF_R4RE, PF_R4IM,
                            PF_PMU, PF_PSCALE, PF_TEMPFAC, PF_POFFSET, PF_MANCHOR, PF_K2, PF_SCATTER};
    for (long long j = 0; j < n; ++j)
        for (int q = 0; q < 24; ++q) o[size_t(j) * 24 + q] = f[size_t(fields[q]) * np + j];
    KS_CUDA(c, cudaMemcpy(out, o.data(), o.size() * sizeof(double), cudaMemcpyDefault));
    return KS_OK;
}

int ks_march_samples(ks_context* c, double* t, double* r, double* theta, double* phi, uint8_t* flags) {
    if (!c || !t || !r || !theta || !phi || !flags) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    KS_CUDA(c, cudaSetDevice(c->device));
    const long long n = c->npix;
    const size_t ns = size_t(n) * c->st.N;
    KS_CUDA(c, c->stage_out.ensure(ns * (4 * sizeof(double) + 1)));
    double* d = c->stage_out.as<double>();
    unsigned char* fl = reinterpret_cast<unsigned char*>(d + 4 * ns);
    KS_CUDA(c, cudaMemsetAsync(d, 0, ns * (4 * sizeof(double) + 1), c->stream));   // samples past a ray's count: zero
    k_march_store<<<nblocks(n), kBlock, 0, c->stream>>>(plan_view(c), c->st, n, d, d + ns, d + 2 * ns, d + 3 * ns, fl,
                                                          c->resid_t.as<double>(), c->resid_phi.as<double>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    KS_CUDA(c, cudaMemcpyAsync(t, d, ns * sizeof(double), cudaMemcpyDefault, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(r, d + ns, ns * sizeof(double), cudaMemcpyDefault, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(theta, d + 2 * ns, ns * sizeof(double), cudaMemcpyDefault, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(phi, d + 3 * ns, ns * sizeof(double), cudaMemcpyDefault, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(flags, fl, ns, cudaMemcpyDefault, c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return KS_OK;
}

int ks_thin_image(ks_context* c, const double* params, int32_t nsplat, double t_obs, int32_t precision, double* out, int32_t order) {
    if (!c || !out) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nsplat < 0 || (nsplat > 0 && !params)) return fail(c, KS_ERR_ARGUMENT, "bad splat count or parameters");
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!std::isfinite(t_obs)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    KS_CUDA(c, cudaSetDevice(c->device));
    const long long n = c->npix;
    const void* dparams = nullptr;
    if (nsplat > 0) {
        int s = stage_in(c, c->stage_in, params, size_t(14) * nsplat * sizeof(double), &dparams);
        if (s) return s;
    }
    KS_CUDA(c, c->tab.ensure(size_t(std::max(nsplat, 1)) * ST_COUNT * sizeof(double)));
    if (nsplat > 0) {
        SetDesc d{KS_THIN14, 14, nsplat, 0, (const double*)dparams, nullptr, 0.0};
        k_splat_table<<<nblocks(nsplat, 64), 64, 0, c->stream>>>(d, c->tab.as<double>());
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    KS_CUDA(c, c->out_sorted.ensure(n * sizeof(double)));
    if (size_t(nsplat) * ST_COUNT * (precision == KS_FP64 ? sizeof(double) : sizeof(float)) > 200 * 1024)
        return fail(c, KS_ERR_ARGUMENT, "too many splats for one launch (%d)", nsplat);
    cudaEventRecord(c->ev0, c->stream);
    int sl = precision == KS_FP64 ? launch_thin<double>(c, c->tab.as<double>(), nsplat, t_obs, nullptr, c->out_sorted.as<double>(), true)
                                  : launch_thin<float>(c, c->tab.as<double>(), nsplat, t_obs, nullptr, c->out_sorted.as<double>(), false);
    if (sl) return sl;
    cudaEventRecord(c->ev1, c->stream);
    int s = emit(c, c->out_sorted.as<double>(), 1, 1, order, out);
    if (s) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->kernel_ms += ms; c->kernel_launches++;
    return KS_OK;
}

int ks_render(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus,
              int32_t nfreq, double L, int32_t precision, int32_t nmax, double slab, double* out, int32_t order) {
    if (!c || !out) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nsets < 0 || (nsets > 0 && !sets)) return fail(c, KS_ERR_ARGUMENT, "bad splat sets");
    if (nframes < 1 || nfreq < 1 || !times || !nus) return fail(c, KS_ERR_ARGUMENT, "need at least one frame and one frequency");
    if (precision != KS_FP64 && precision != KS_MIXED && precision != KS_MIXED_GEO64)
        return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!(std::isfinite(L) && L > 0)) return fail(c, KS_ERR_NONFINITE, "length unit must be finite and positive");
    c->geo64 = precision == KS_MIXED_GEO64;
    if (precision == KS_MIXED_GEO64) precision = KS_MIXED;
    if (!std::isfinite(slab)) return fail(c, KS_ERR_NONFINITE, "non-finite slab");
    KS_CUDA(c, cudaSetDevice(c->device));
    std::vector<double> ht(nframes), hnu(nfreq);
    KS_CUDA(c, cudaMemcpy(ht.data(), times, nframes * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(hnu.data(), nus, nfreq * sizeof(double), cudaMemcpyDefault));
    for (double v : ht) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    for (double v : hnu) if (!(std::isfinite(v) && v > 0)) return fail(c, KS_ERR_NONFINITE, "frequencies must be finite and positive");
    int ntot = 0;
    {
        int st_ = build_tables(c, sets, nsets, &ntot, false);
        if (st_) return st_;
    }
    const long long n = c->npix;
    const int ncombo = nframes * nfreq;
    std::vector<double> hc(ht);   // times then frequencies
    hc.insert(hc.end(), hnu.begin(), hnu.end());
    // sized for the adjoint's layout too (times, frequencies, then per combination), so that an
    // adjoint call does not move the buffer under a captured render
    KS_CUDA(c, c->combos.ensure((size_t(nframes) + nfreq + 2 * size_t(ncombo)) * sizeof(double)));
    KS_CUDA(c, cudaMemcpyAsync(c->combos.p, hc.data(), hc.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    KS_CUDA(c, c->out_sorted.ensure(size_t(n) * 4 * ncombo * sizeof(double)));
    if (c->count_events) {
        KS_CUDA(c, c->counters.ensure(8 * sizeof(unsigned long long)));
        KS_CUDA(c, cudaMemsetAsync(c->counters.p, 0, 8 * sizeof(unsigned long long), c->stream));
    }
    cudaEventRecord(c->ev0, c->stream);
    bool thermal_only = true;
    for (int q = 0; q < nsets; ++q) thermal_only = thermal_only && (sets[q].kind == KS_THERMAL21 || sets[q].nsplat == 0);
    if (precision == KS_FP64 && (size_t(ntot) * ST_COUNT + c->nkv) * sizeof(double) > 220 * 1024)
        return fail(c, KS_ERR_ARGUMENT, "too many splats for one launch (%d)", ntot);
    int sl = precision == KS_FP64 ? launch_plain(c, ntot, nframes, nfreq, L, nmax, slab, thermal_only)
                                  : launch_mixed(c, ntot, nframes, nfreq, L, nmax, slab, thermal_only);
    if (sl) return sl;
    cudaEventRecord(c->ev1, c->stream);
    KS_CUDA(c, cudaGetLastError());
    int s = emit(c, c->out_sorted.as<double>(), 4, ncombo, order, out);
    if (s) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->kernel_ms += ms;
    if (precision != KS_FP64 && c->consume_timed) {
        float mc = 0.f;
        cudaEventElapsedTime(&mc, c->evc0, c->evc1);
        c->consume_ms += mc;
        c->consume_launches++;
        c->consume_timed = false;
    }
    return check_device_flag(c, "ks_render");
}

int ks_riaf_image(ks_context* c, const double* model, int32_t pandya, const double* nus, int32_t nfreq, double L, int32_t precision,
                  double* out, int32_t order) {
    if (!c || !out || !model || !nus) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nfreq < 1) return fail(c, KS_ERR_ARGUMENT, "need at least one frequency");
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!(std::isfinite(L) && L > 0)) return fail(c, KS_ERR_NONFINITE, "length unit must be finite and positive");
    KS_CUDA(c, cudaSetDevice(c->device));
    double hm[KS_RIAF_PARAMS];
    KS_CUDA(c, cudaMemcpy(hm, model, sizeof hm, cudaMemcpyDefault));
    for (double v : hm) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite RIAF parameter");
    if (!(hm[9] > 0 && hm[8] > 0 && hm[2] > 0)) return fail(c, KS_ERR_ARGUMENT, "RIAF needs positive disk_h, r_isco and rout");
    std::vector<double> hnu(nfreq);
    KS_CUDA(c, cudaMemcpy(hnu.data(), nus, nfreq * sizeof(double), cudaMemcpyDefault));
    for (double v : hnu) if (!(std::isfinite(v) && v > 0)) return fail(c, KS_ERR_NONFINITE, "frequencies must be finite and positive");
    const RiafModel m{hm[0], hm[1], hm[2], hm[3], hm[4], hm[5], hm[6], hm[7], hm[8], hm[9], pandya != 0};
    const long long n = c->npix;
    KS_CUDA(c, c->combos.ensure(hnu.size() * sizeof(double)));
    KS_CUDA(c, cudaMemcpyAsync(c->combos.p, hnu.data(), hnu.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    KS_CUDA(c, c->out_sorted.ensure(size_t(n) * 4 * nfreq * sizeof(double)));
    if (c->count_events) {
        KS_CUDA(c, c->counters.ensure(8 * sizeof(unsigned long long)));
        KS_CUDA(c, cudaMemsetAsync(c->counters.p, 0, 8 * sizeof(unsigned long long), c->stream));
    }
    unsigned long long* ctr = c->count_events ? c->counters.as<unsigned long long>() : nullptr;
    cudaEventRecord(c->ev0, c->stream);
    const dim3 grid(unsigned(nblocks(n)), unsigned(nfreq));
    if (precision == KS_FP64)
        k_riaf<double><<<grid, kBlock, 0, c->stream>>>(plan_view(c), c->st, n, m, c->combos.as<double>(), L, c->out_sorted.as<double>(), ctr);
    else
        k_riaf<float><<<grid, kBlock, 0, c->stream>>>(plan_view(c), c->st, n, m, c->combos.as<double>(), L, c->out_sorted.as<double>(), ctr);
    cudaEventRecord(c->ev1, c->stream);
    c->launches++;
    c->kernel_launches++;
    KS_CUDA(c, cudaGetLastError());
    int s = emit(c, c->out_sorted.as<double>(), 4, nfreq, order, out);
    if (s) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->kernel_ms += ms;
    return KS_OK;
}

// The device buffers a captured render reads or writes (a replay requires them unmoved).
std::vector<void*> graph_buffers(const ks_context* c) {
    return {c->rows.p, c->kstop.p, c->stream_buf.p, c->seg_out.p, c->work.p, c->out_sorted.p, c->errflag.p, c->perm.p, c->plan.p,
            c->anchors.p, c->aoff.p};
}

void release_graph(cudaGraph_t& g, cudaGraphExec_t& ex) {
    if (ex) cudaGraphExecDestroy(ex);
    if (g) cudaGraphDestroy(g);
    ex = nullptr;
    g = nullptr;
}

// ... and those of a captured chi^2 + gradient evaluation
std::vector<void*> chi2_graph_buffers(const ks_context* c) {
    std::vector<void*> b = graph_buffers(c);
    for (const DevBuf* d : {&c->gtab, &c->adj_state, &c->adj_act, &c->adj_bnd, &c->adj_unit, &c->adj_part, &c->seeds, &c->chi_part,
                            &c->chi_val, &c->dgrad})
        b.push_back(d->p);
    return b;
}

// A capture's own copies of its call's splat table (whose knots stay as they are) and of its times and frequencies: every
// later call writes its own into the context's buffers. In the context's place while it exists.
struct GraphInputs {
    ks_context* c;
    DevBuf &tab, &combos;
    GraphInputs(ks_context* c_, DevBuf& t, DevBuf& s) : c(c_), tab(t), combos(s) { c->tab.swap(tab); c->combos.swap(combos); }
    ~GraphInputs() { c->tab.swap(tab); c->combos.swap(combos); }
};
int copy_graph_inputs(ks_context* c, DevBuf& tab, DevBuf& combos, int ntot, int nframes, int nfreq) {
    const size_t nt = (size_t(std::max(ntot, 1)) * ST_COUNT + c->nkv) * sizeof(double), nc = (size_t(nframes) + nfreq) * sizeof(double);
    KS_CUDA(c, tab.ensure(nt));
    KS_CUDA(c, combos.ensure(nc));
    KS_CUDA(c, cudaMemcpyAsync(tab.p, c->tab.p, nt, cudaMemcpyDeviceToDevice, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(combos.p, c->combos.p, nc, cudaMemcpyDeviceToDevice, c->stream));
    return KS_OK;
}

// The splat tables of device-resident sets rebuilt on the device inside a capture (the knot array
// stays as the ordinary call before the capture wrote it): k_splat_table per set, with grad the
// gradient table (k_grad_table).
int capture_tables(ks_context* c, const ks_splat_set* sets, int nsets, int ntot, bool grad) {
    int first = 0, koff = 0;
    for (int s = 0; s < nsets; ++s) {
        const ks_splat_set& S = sets[s];
        if (S.nsplat == 0) continue;
        const int nk = S.kind == KS_KNOT21 ? S.nknots : 0;
        SetDesc d{S.kind, nrows_of(S.kind), S.nsplat, first, static_cast<const double*>(S.params),
                  S.kind == KS_KAPPA22 ? static_cast<const double*>(S.hyp) : nullptr, S.gamma_max > 0 ? S.gamma_max : 1e5,
                  S.kind == KS_KNOT21 ? koff : 0, nk,
                  c->tab.as<const double>() + size_t(ntot) * ST_COUNT};
        k_splat_table<<<nblocks(S.nsplat, 64), 64, 0, c->stream>>>(d, c->tab.as<double>());
        if (grad) k_grad_table<<<nblocks(S.nsplat, 64), 64, 0, c->stream>>>(S.nsplat, first, static_cast<const double*>(S.params),
                                                                           c->gtab.as<double>());
        if (cudaGetLastError() != cudaSuccess) return fail(c, KS_ERR_DEVICE, "graph capture: splat table of set %d", s);
        first += S.nsplat;
        koff += S.nsplat * 4 * nk;   // per knot splat: its nk times and 3 nk centres
    }
    return KS_OK;
}

// One mixed render of device-resident splat sets recorded into a CUDA graph: the splat tables built
// from the parameters (in place on the device), the sample stream, the transport, the
// segment composition and the output in `order`. Frames, frequencies, L, the knot array, the splat
// counts and the pointers are fixed at capture; a replay re-reads the parameter values.
int ks_render_graph_capture(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes,
                            const double* nus, int32_t nfreq, double L, int32_t nmax, double slab, double* out, int32_t order) {
    if (!c || !out || !sets || nsets < 1) return KS_ERR_ARGUMENT;
    if (!is_device_ptr(out)) return fail(c, KS_ERR_ARGUMENT, "the graph's output must be device memory");
    for (int s = 0; s < nsets; ++s) {
        if (sets[s].nsplat > 0 && !is_device_ptr(sets[s].params))
            return fail(c, KS_ERR_ARGUMENT, "set %d: a graph reads device-resident parameters", s);
        if (sets[s].kind == KS_KAPPA22 && sets[s].nsplat > 0 && !is_device_ptr(sets[s].hyp))
            return fail(c, KS_ERR_ARGUMENT, "set %d: a graph reads device-resident hyp", s);
    }
    release_graph(c->graph, c->graph_exec);
    const bool counting = c->count_events;
    c->count_events = false;
    // one ordinary render: validation, tables and knots, buffers, the launch shape
    int status = ks_render(c, sets, nsets, times, nframes, nus, nfreq, L, KS_MIXED, nmax, slab, out, order);
    c->count_events = counting;
    if (status) return status;
    int ntot = 0;
    bool thermal_only = true;
    for (int s = 0; s < nsets; ++s) {
        ntot += sets[s].nsplat;
        thermal_only = thermal_only && (sets[s].kind == KS_THERMAL21 || sets[s].nsplat == 0);
    }
    if ((status = copy_graph_inputs(c, c->graph_tab, c->graph_combos, ntot, nframes, nfreq))) return status;
    GraphInputs own(c, c->graph_tab, c->graph_combos);
    KS_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
    c->capturing = true;
    status = capture_tables(c, sets, nsets, ntot, false);
    if (status == KS_OK) status = launch_mixed(c, ntot, nframes, nfreq, L, nmax, slab, thermal_only);
    if (status == KS_OK) status = emit(c, c->out_sorted.as<double>(), 4, nframes * nfreq, order, out);
    cudaGraph_t g = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(c->stream, &g);
    c->capturing = false;
    if (status != KS_OK || ec != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        return status != KS_OK ? status : fail(c, KS_ERR_DEVICE, "graph capture: %s", cudaGetErrorString(ec));
    }
    cudaGraphExec_t ex = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&ex, g, 0);
    if (ei != cudaSuccess) {
        cudaGraphDestroy(g);
        cudaGetLastError();
        return fail(c, KS_ERR_DEVICE, "graph instantiation: %s", cudaGetErrorString(ei));
    }
    c->graph = g;
    c->graph_exec = ex;
    c->graph_bufs = graph_buffers(c);
    return KS_OK;
}

// Replay the captured render on the context stream; with wait, synchronise and report a kernel whose
// bounded wait gave up.
int ks_graph_launch(ks_context* c, int32_t wait) {
    if (!c) return KS_ERR_ARGUMENT;
    if (!c->graph_exec) return fail(c, KS_ERR_ARGUMENT, "no captured graph");
    if (graph_buffers(c) != c->graph_bufs)
        return fail(c, KS_ERR_ARGUMENT, "a later call reallocated buffers the graph uses: capture again");
    KS_CUDA(c, cudaGraphLaunch(c->graph_exec, c->stream));
    c->launches++;
    if (!wait) return KS_OK;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_device_flag(c, "graph replay");
}

int ks_graph_destroy(ks_context* c) {
    if (!c) return KS_ERR_ARGUMENT;
    release_graph(c->graph, c->graph_exec);
    release_graph(c->cgraph, c->cgraph_exec);
    for (DevBuf* d : {&c->graph_tab, &c->graph_combos, &c->cgraph_tab, &c->cgraph_combos}) d->release();
    return KS_OK;
}

}  // extern "C"

// ---- the adjoint (src/Splats/dual_gradient.jl, src/Fit/Fit.jl:451-577) --------------------------------

namespace {
int gemm(ks_context* c, int M, int N, int K, const float* Ah, const float* Al, long long lda, const float* Bh, const float* Bl, long long ldb,
         float* C, long long ldc);
int dft_stage(ks_context* c, int slot, const double* src, size_t count, const double** dev);
int dft_checks(ks_context* c, int64_t nuv, double psize, double scale, int32_t precision);
int dft_forward(ks_context* c, const double* dimg, int32_t order, int64_t nuv, const double* du, const double* dv, const double* dtap,
                double psize, double scale, int32_t precision, double* dV);
int dft_adjoint(ks_context* c, const double* dw, int64_t nuv, const double* du, const double* dv, const double* dtap, double psize,
                double scale, int32_t precision, double* dseed, int32_t order, bool have_twiddles);

// The visibility data of a frame (frame_chi2_seed!, device_visibilities.jl:97-111): nuv baselines,
// the gains g (complex, may be NULL), the data vis and sigma per Stokes; all host or device.
struct VisData {
    int64_t nuv;
    const double *u, *v, *tap, *g, *vis, *sigma;
    double psize, scale;
};
}

namespace {

// dst is left as it was when a kernel before it gave up (`err`: the device flag)
__global__ void k_accumulate(double* __restrict__ dst, const double* __restrict__ src, long long n, int accumulate, const unsigned* __restrict__ err) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q < n && *err == 0u) dst[q] = (accumulate ? dst[q] : 0.0) + src[q];
}

// Stage `count` elements of `src` (host or device) into `buf`; returns the device pointer.
template <class U>
int stage_dev(ks_context* c, DevBuf& buf, const U* src, size_t count, const U** dev) {
    if (!src) { *dev = nullptr; return KS_OK; }
    const void* d = nullptr;
    int s = stage_in(c, buf, src, count * sizeof(U), &d);
    *dev = reinterpret_cast<const U*>(d);
    return s;
}

// The forward and the reverse pass of a gradient, the state of `piece` rays at a time. With the state of every ray held,
// the forward pass leaves it; else the forward pass is the image alone and the reverse pass goes over the screen piece by
// piece. Pieces are halved while memory runs out (`fixed`: not in a capture, which takes the piece of the call before it).
struct GradientPasses {
    ks_context* c;
    int ntot, nframes, nfreq, nmax;
    double L, slab;
    bool plain, fixed;
    long long piece;
    bool shrink(int s) {
        if (s != KS_ERR_OUT_OF_MEMORY || fixed || piece <= 32) return false;
        release_state(c);
        piece = smaller_piece(piece);
        return true;
    }
    int state(long long j0) { return launch_state(c, plain, ntot, nframes, nfreq, L, nmax, slab, j0, std::min(piece, c->npix - j0), piece); }
    int forward() {
        int s = KS_OK;
        do
            s = piece >= c->npix ? state(0) : plain ? launch_plain(c, ntot, nframes, nfreq, L, nmax, slab, true)
                                                    : launch_mixed(c, ntot, nframes, nfreq, L, nmax, slab, true);
        while (shrink(s));
        return s;
    }
    int reverse() {
        for (long long j0 = 0; ntot > 0 && j0 < c->npix;) {
            int s = piece < c->npix ? state(j0) : KS_OK;
            if (s == KS_OK) s = launch_reverse(c, ntot, nmax, plain, j0 > 0);
            if (shrink(s)) { j0 = 0; continue; }
            if (s) return s;
            j0 += piece;
        }
        c->state_piece = piece;
        return KS_OK;
    }
};

// The forward image, the seeds (given, or those of chi^2), the reverse pass and the reduction into dparams.
int adjoint_run(ks_context* c, const ks_splat_set* sets, int nsets, const double* times, int nframes, const double* nus, int nfreq,
                double L, int precision, int nmax, double slab, const double* dstokes, int order, const double* data,
                const double* sigma, double sigma_s, const uint8_t* mask, double* chi2_out, double* dparams, int accumulate,
                double* image, const VisData* vd = nullptr) {
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nsets < 0 || (nsets > 0 && !sets)) return fail(c, KS_ERR_ARGUMENT, "bad splat sets");
    if (nframes < 1 || nfreq < 1 || !times || !nus) return fail(c, KS_ERR_ARGUMENT, "need at least one frame and one frequency");
    const bool geo = precision == KS_MIXED_GEO64;   // the FP64 march under the mixed transport
    if (geo) precision = KS_MIXED;
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d for the adjoint", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!(std::isfinite(L) && L > 0)) return fail(c, KS_ERR_NONFINITE, "length unit must be finite and positive");
    if (!std::isfinite(slab)) return fail(c, KS_ERR_NONFINITE, "non-finite slab");
    if (!dparams) return fail(c, KS_ERR_ARGUMENT, "dparams is required");
    if (data && !sigma && !(std::isfinite(sigma_s) && sigma_s > 0))
        return fail(c, KS_ERR_ARGUMENT, "chi^2 needs sigma (an array, or a finite positive scalar)");
    KS_CUDA(c, cudaSetDevice(c->device));
    std::vector<double> ht(nframes), hnu(nfreq);
    KS_CUDA(c, cudaMemcpy(ht.data(), times, nframes * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(hnu.data(), nus, nfreq * sizeof(double), cudaMemcpyDefault));
    for (double v : ht) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    for (double v : hnu) if (!(std::isfinite(v) && v > 0)) return fail(c, KS_ERR_NONFINITE, "frequencies must be finite and positive");
    int ntot = 0;
    {
        int s = build_tables(c, sets, nsets, &ntot, true);
        if (s) return s;
    }
    const long long n = c->npix;
    const int N = c->st.N;
    const int ncombo = nframes * nfreq;
    const long long nrc = n * ncombo;
    std::vector<double> hc(ht);   // the times, then the frequencies
    hc.insert(hc.end(), hnu.begin(), hnu.end());
    KS_CUDA(c, c->combos.ensure((size_t(nframes) + nfreq + 2 * size_t(ncombo)) * sizeof(double)));
    KS_CUDA(c, cudaMemcpyAsync(c->combos.p, hc.data(), hc.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    KS_CUDA(c, c->out_sorted.ensure(size_t(nrc) * 4 * sizeof(double)));
    KS_CUDA(c, c->seeds.ensure(size_t(nrc) * 4 * sizeof(double)));
    KS_CUDA(c, c->dgrad.ensure(size_t(std::max(ntot, 1)) * GR_COUNT * sizeof(double)));
    cudaEventRecord(c->ev0, c->stream);
    const bool mixed = precision == KS_MIXED;
    // 1. forward pass with the reverse pass's state
    if (mixed) c->geo64 = geo;
    else if (size_t(ntot) * ST_COUNT * sizeof(double) > 200 * 1024) return fail(c, KS_ERR_ARGUMENT, "too many splats for the FP64 adjoint (%d)", ntot);
    GradientPasses passes{c, ntot, nframes, nfreq, nmax, L, slab, !mixed, false, state_rays(c, !mixed, nframes, nfreq)};
    if (int s = passes.forward()) return s;
    // 2. seeds
    const long long nblk = (nrc + 255) / 256;
    double vis_chi2 = 0.0;
    if (vd) {
        // the visibilities of the image, chi^2 of the gained model and the adjoint transform of its
        // weights (frame_chi2_seed!): the DFT in the render's precision class (3xTF32 for the mixed path)
        if (ncombo != 1) return fail(c, KS_ERR_ARGUMENT, "visibility chi^2 takes one frame at one frequency");
        const int dprec = mixed ? KS_MIXED : KS_FP64;
        int s = dft_checks(c, vd->nuv, vd->psize, vd->scale, dprec);
        if (s) return s;
        const int64_t nuv = vd->nuv;
        const double *du, *dv, *dtap, *dg, *dvis;
        if ((s = dft_stage(c, 1, vd->u, nuv, &du)) || (s = dft_stage(c, 2, vd->v, nuv, &dv)) ||
            (s = dft_stage(c, 3, vd->tap, vd->tap ? nuv : 0, &dtap)) || (s = dft_stage(c, 6, vd->g, vd->g ? 2 * nuv : 0, &dg)) ||
            (s = dft_stage(c, 7, vd->vis, size_t(nuv) * 8, &dvis)))
            return s;
        KS_CUDA(c, c->dft_in[4].ensure(size_t(nuv) * 8 * sizeof(double) * 2 + size_t(nuv) * 4 * sizeof(double)));
        double* dV = c->dft_in[4].as<double>();
        double* dW = dV + nuv * 8;
        double* dS = dW + nuv * 8;
        KS_CUDA(c, cudaMemcpyAsync(dS, vd->sigma, size_t(nuv) * 4 * sizeof(double), cudaMemcpyDefault, c->stream));
        if ((s = dft_forward(c, c->out_sorted.as<double>(), KS_ORDER_SORTED, nuv, du, dv, dtap, vd->psize, vd->scale, dprec, dV))) return s;
        const int vblk = int((nuv * 4 + 255) / 256);
        KS_CUDA(c, c->dft_partial.ensure(size_t(vblk) * sizeof(double)));
        ksdft::k_chi2_weights<<<vblk, 256, 0, c->stream>>>(nuv, dV, dg, dvis, dS, dW, c->dft_partial.as<double>());
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
        if ((s = dft_adjoint(c, dW, nuv, du, dv, dtap, vd->psize, vd->scale, dprec, c->seeds.as<double>(), KS_ORDER_SORTED, dprec != KS_FP64)))
            return s;
        std::vector<double> part(vblk);
        KS_CUDA(c, cudaMemcpyAsync(part.data(), c->dft_partial.p, vblk * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        KS_CUDA(c, cudaStreamSynchronize(c->stream));
        for (double p : part) vis_chi2 += p;   // fixed order
    } else if (data) {
        const double *dd = nullptr, *ds = nullptr;
        const uint8_t* dm = nullptr;
        KS_CUDA(c, c->dstage.ensure(size_t(nrc) * 4 * sizeof(double) * (sigma ? 2 : 1) + size_t(nrc)));
        // host data, sigma and mask share one staging buffer
        const bool hd = !is_device_ptr(data), hs = sigma && !is_device_ptr(sigma), hm = mask && !is_device_ptr(mask);
        double* st0 = c->dstage.as<double>();
        if (hd) { KS_CUDA(c, cudaMemcpyAsync(st0, data, size_t(nrc) * 4 * sizeof(double), cudaMemcpyHostToDevice, c->stream)); dd = st0; }
        else dd = data;
        if (sigma) {
            if (hs) { KS_CUDA(c, cudaMemcpyAsync(st0 + nrc * 4, sigma, size_t(nrc) * 4 * sizeof(double), cudaMemcpyHostToDevice, c->stream)); ds = st0 + nrc * 4; }
            else ds = sigma;
        }
        if (mask) {
            uint8_t* m0 = reinterpret_cast<uint8_t*>(st0 + nrc * 4 * (sigma ? 2 : 1));
            if (hm) { KS_CUDA(c, cudaMemcpyAsync(m0, mask, size_t(nrc), cudaMemcpyHostToDevice, c->stream)); dm = m0; }
            else dm = mask;
        }
        KS_CUDA(c, c->chi_part.ensure(size_t(nblk) * sizeof(double)));
        KS_CUDA(c, c->chi_val.ensure(sizeof(double)));
        k_chi2_seed<<<unsigned(nblk), 256, 0, c->stream>>>(c->out_sorted.as<double>(), c->perm.as<long long>(), n, ncombo, dd, ds, sigma_s, dm,
                                                           c->seeds.as<double>(), c->chi_part.as<double>());
        k_sum_partials<<<1, 256, 0, c->stream>>>(c->chi_part.as<double>(), nblk, c->chi_val.as<double>());
        c->launches += 2;
        KS_CUDA(c, cudaGetLastError());
    } else {
        const double* dsd = nullptr;
        {
            int s = stage_dev(c, c->dstage, dstokes, size_t(nrc) * 4, &dsd);
            if (s) return s;
        }
        k_sort_seed<<<nblocks(nrc, 256), 256, 0, c->stream>>>(dsd, c->perm.as<long long>(), n, ncombo, order == KS_ORDER_SCREEN ? 1 : 0,
                                                              c->seeds.as<double>());
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    // 3. reverse pass and the deterministic reduction
    if (int s = passes.reverse()) return s;
    cudaEventRecord(c->ev1, c->stream);
    // 4. results; the gradient only if no kernel gave up
    const long long ng = (long long)ntot * GR_COUNT;
    std::vector<double> hg;
    if (ng > 0) {
        if (is_device_ptr(dparams)) {
            k_accumulate<<<nblocks(ng, 256), 256, 0, c->stream>>>(dparams, c->dgrad.as<double>(), ng, accumulate, c->errflag.as<unsigned>());
            c->launches++;
            KS_CUDA(c, cudaGetLastError());
        } else {
            hg.resize(ng);
            KS_CUDA(c, cudaMemcpyAsync(hg.data(), c->dgrad.p, ng * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        }
    }
    if (data && chi2_out) KS_CUDA(c, cudaMemcpyAsync(chi2_out, c->chi_val.p, sizeof(double), cudaMemcpyDefault, c->stream));
    if (vd && chi2_out) *chi2_out = vis_chi2;
    if (image) {
        int s = emit(c, c->out_sorted.as<double>(), 4, ncombo, KS_ORDER_SCREEN, image);
        if (s) return s;
    }
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->adjoint_ms += ms;
    const int flag = check_device_flag(c, "adjoint");
    if (flag) return flag;
    for (size_t q = 0; q < hg.size(); ++q) dparams[q] = (accumulate ? dparams[q] : 0.0) + hg[q];
    return KS_OK;
}

}  // namespace

extern "C" {

int ks_adjoint(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus,
               int32_t nfreq, double L, int32_t precision, int32_t nmax, double slab, const double* dstokes, int32_t order,
               double* dparams, int32_t accumulate) {
    if (!c || !dstokes) return KS_ERR_ARGUMENT;
    return adjoint_run(c, sets, nsets, times, nframes, nus, nfreq, L, precision, nmax, slab, dstokes, order, nullptr, nullptr, 0.0,
                       nullptr, nullptr, dparams, accumulate, nullptr);
}

int ks_chi2_gradient(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus,
                     int32_t nfreq, double L, int32_t precision, int32_t nmax, double slab, const double* data, const double* sigma,
                     double sigma_scalar, const uint8_t* mask, double* chi2, double* dparams, int32_t accumulate, double* image) {
    if (!c || !data) return KS_ERR_ARGUMENT;
    return adjoint_run(c, sets, nsets, times, nframes, nus, nfreq, L, precision, nmax, slab, nullptr, KS_ORDER_SCREEN, data, sigma,
                       sigma_scalar, mask, chi2, dparams, accumulate, image);
}

// One mixed chi^2 + gradient evaluation of device-resident thermal sets against device-resident
// image-domain data, recorded into a CUDA graph: the splat and gradient tables from the parameters,
// the sample stream, the forward pass with the reverse pass's state, chi^2 and its seeds, the reverse
// pass, the fixed-order reduction into dparams, chi^2 into `chi2`. It runs one ordinary evaluation
// first (validation, buffers, launch shapes), which writes chi2 and dparams as ks_chi2_gradient does.
int ks_chi2_gradient_graph_capture(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes,
                                   const double* nus, int32_t nfreq, double L, int32_t nmax, double slab, const double* data,
                                   const double* sigma, double sigma_scalar, const uint8_t* mask, double* chi2, double* dparams,
                                   int32_t accumulate) {
    if (!c || !sets || nsets < 1 || !data || !chi2 || !dparams) return KS_ERR_ARGUMENT;
    if (!is_device_ptr(data) || (sigma && !is_device_ptr(sigma)) || (mask && !is_device_ptr(mask)) || !is_device_ptr(chi2) ||
        !is_device_ptr(dparams))
        return fail(c, KS_ERR_ARGUMENT, "a captured chi^2 + gradient reads and writes device memory only (data, sigma, mask, chi2, dparams)");
    for (int s = 0; s < nsets; ++s)
        if (sets[s].nsplat > 0 && !is_device_ptr(sets[s].params))
            return fail(c, KS_ERR_ARGUMENT, "set %d: a graph reads device-resident parameters", s);
    release_graph(c->cgraph, c->cgraph_exec);
    const bool counting = c->count_events;
    c->count_events = false;
    int status = adjoint_run(c, sets, nsets, times, nframes, nus, nfreq, L, KS_MIXED, nmax, slab, nullptr, KS_ORDER_SCREEN, data, sigma,
                             sigma_scalar, mask, chi2, dparams, accumulate, nullptr);
    c->count_events = counting;
    if (status) return status;
    int ntot = 0;
    for (int s = 0; s < nsets; ++s) ntot += sets[s].nsplat;
    const long long n = c->npix;
    const int ncombo = nframes * nfreq;
    const long long nrc = n * ncombo;
    const long long nblk = (nrc + 255) / 256;
    if ((status = copy_graph_inputs(c, c->cgraph_tab, c->cgraph_combos, ntot, nframes, nfreq))) return status;
    GraphInputs own(c, c->cgraph_tab, c->cgraph_combos);
    KS_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
    c->capturing = true;
    status = capture_tables(c, sets, nsets, ntot, true);
    c->geo64 = false;
    GradientPasses passes{c, ntot, nframes, nfreq, nmax, L, slab, false, true, c->state_piece};
    if (status == KS_OK) status = passes.forward();
    if (status == KS_OK) {
        k_chi2_seed<<<unsigned(nblk), 256, 0, c->stream>>>(c->out_sorted.as<double>(), c->perm.as<long long>(), n, ncombo, data, sigma,
                                                           sigma_scalar, mask, c->seeds.as<double>(), c->chi_part.as<double>());
        k_sum_partials<<<1, 256, 0, c->stream>>>(c->chi_part.as<double>(), nblk, c->chi_val.as<double>());
        if (cudaGetLastError() != cudaSuccess) status = fail(c, KS_ERR_DEVICE, "graph capture: chi^2 seeds");
    }
    if (status == KS_OK) status = passes.reverse();
    const long long ng = (long long)ntot * GR_COUNT;
    if (status == KS_OK && ng > 0) {
        k_accumulate<<<nblocks(ng, 256), 256, 0, c->stream>>>(dparams, c->dgrad.as<double>(), ng, accumulate, c->errflag.as<unsigned>());
        if (cudaGetLastError() != cudaSuccess) status = fail(c, KS_ERR_DEVICE, "graph capture: gradient");
    }
    if (status == KS_OK && cudaMemcpyAsync(chi2, c->chi_val.p, sizeof(double), cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess)
        status = fail(c, KS_ERR_DEVICE, "graph capture: chi^2");
    cudaGraph_t g = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(c->stream, &g);
    c->capturing = false;
    if (status != KS_OK || ec != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        return status != KS_OK ? status : fail(c, KS_ERR_DEVICE, "graph capture: %s", cudaGetErrorString(ec));
    }
    cudaGraphExec_t ex = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&ex, g, 0);
    if (ei != cudaSuccess) {
        cudaGraphDestroy(g);
        cudaGetLastError();
        return fail(c, KS_ERR_DEVICE, "graph instantiation: %s", cudaGetErrorString(ei));
    }
    c->cgraph = g;
    c->cgraph_exec = ex;
    c->cgraph_bufs = chi2_graph_buffers(c);
    return KS_OK;
}

// Replay the captured chi^2 + gradient evaluation on the context stream; with wait, synchronise and
// report a kernel whose bounded wait gave up.
int ks_chi2_gradient_graph_launch(ks_context* c, int32_t wait) {
    if (!c) return KS_ERR_ARGUMENT;
    if (!c->cgraph_exec) return fail(c, KS_ERR_ARGUMENT, "no captured chi^2 + gradient graph");
    if (chi2_graph_buffers(c) != c->cgraph_bufs)
        return fail(c, KS_ERR_ARGUMENT, "a later call reallocated buffers the graph uses: capture again");
    KS_CUDA(c, cudaGraphLaunch(c->cgraph_exec, c->stream));
    c->launches++;
    if (!wait) return KS_OK;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return check_device_flag(c, "chi^2 + gradient graph replay");
}

}  // extern "C"

namespace {

// J v of the image for one chunk of K directions (dirs: K x nparams, each laid out like dparams)
template <class S, int K>
int jvp_chunk(ks_context* c, int ntot, const double* dparams_dev, const double* ddirs, long long dstride, const double* dct,
              const double* dcn, int ncombo, double L, int nmax, double slab, double* img_sorted, double* out_sorted, int lnL_dir = -1) {
    KS_CUDA(c, c->jvp_tab.ensure(size_t(std::max(ntot, 1)) * ST_COUNT * sizeof(Dual<S, K>)));
    Dual<S, K>* dt = c->jvp_tab.as<Dual<S, K>>();
    if (ntot > 0) {
        k_dual_table<S, K><<<nblocks(ntot, 64), 64, 0, c->stream>>>(ntot, dparams_dev, ddirs, dstride, c->tab.as<double>(),
                                                                    c->gtab.as<double>(), dt);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    const long long nrc = c->npix * ncombo;
    if constexpr (std::is_same<S, float>::value) {
        // segments until there are some 32 warps per SM (at least 16 samples each), as far as 4 GB of segment states go
        int nseg = 1;
        while (nrc * nseg < c->nsm * 1024LL && (nseg * 2) * 16 <= c->st.N && nrc * nseg * 2 * 20 * (K + 1) * (long long)sizeof(float) <= (4LL << 30)) nseg *= 2;
        // fewer where memory runs out
        for (;; nseg /= 2) {
            const cudaError_t e = c->jvp_part.ensure(size_t(nrc) * nseg * 20 * (K + 1) * sizeof(float));
            if (e == cudaErrorMemoryAllocation && nseg > 1) { cudaGetLastError(); continue; }
            KS_CUDA(c, e);
            break;
        }
        const int seg_len = (c->st.N + nseg - 1) / nseg;
        const int* kstop = nullptr;
        if (nmax >= 0) {
            int s = launch_wind_stop(c, nmax, slab);
            if (s) return s;
            kstop = c->kstop.as<int>();
        }
        k_jvp_stream<K><<<nblocks(nrc * nseg, 64), 64, 0, c->stream>>>(plan_view(c), c->st, c->npix, dt, ntot, dct, dcn, ncombo, L, kstop, nseg, seg_len,
                                                                       c->stream_buf.as<float>(), c->jvp_part.as<float>(), lnL_dir);
        k_jvp_combine<K><<<nblocks(nrc, 128), 128, 0, c->stream>>>(c->npix, ncombo, nseg, dcn, c->jvp_part.as<float>(), img_sorted, out_sorted);
        c->launches++;
    } else
        k_jvp<S, K><<<nblocks(nrc, 64), 64, 0, c->stream>>>(plan_view(c), c->st, c->npix, dt, ntot, dct, dcn, ncombo, L, nmax, slab, img_sorted,
                                                            out_sorted, lnL_dir);
    c->launches++;
    c->adjoint_launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

}  // namespace

extern "C" {

}  // extern "C"

namespace {

// ks_jvp; with lnL, one direction: d/d(ln L) (dirs ignored), exact through a dual step length
int jvp_impl(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus, int32_t nfreq,
             double L, int32_t precision, int32_t nmax, double slab, const double* dirs, int32_t ndir, double* dimage, int32_t order,
             double* image, bool lnL) {
    if (!c || (!dirs && !lnL) || !dimage || ndir < 1) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nsets < 1 || !sets) return fail(c, KS_ERR_ARGUMENT, "bad splat sets");
    if (nframes < 1 || nfreq < 1 || !times || !nus) return fail(c, KS_ERR_ARGUMENT, "need at least one frame and one frequency");
    const bool geo = precision == KS_MIXED_GEO64;
    if (geo) precision = KS_MIXED;
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d for the JVP", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!(std::isfinite(L) && L > 0)) return fail(c, KS_ERR_NONFINITE, "length unit must be finite and positive");
    KS_CUDA(c, cudaSetDevice(c->device));
    std::vector<double> ht(nframes), hnu(nfreq);
    KS_CUDA(c, cudaMemcpy(ht.data(), times, nframes * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(hnu.data(), nus, nfreq * sizeof(double), cudaMemcpyDefault));
    for (double v : ht) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    for (double v : hnu) if (!(std::isfinite(v) && v > 0)) return fail(c, KS_ERR_NONFINITE, "frequencies must be finite and positive");
    int ntot = 0;
    {
        int s = build_tables(c, sets, nsets, &ntot, true);
        if (s) return s;
    }
    // the raw parameters of all sets, concatenated (21 x ntot) on the device
    const long long np = (long long)ntot * 21;
    std::vector<double> hp(np);
    {
        long long off = 0;
        for (int s = 0; s < nsets; ++s) {
            const size_t cnt = size_t(21) * sets[s].nsplat;
            if (cnt) KS_CUDA(c, cudaMemcpy(hp.data() + off, sets[s].params, cnt * sizeof(double), cudaMemcpyDefault));
            off += cnt;
        }
    }
    // directions of a pass: the FP32 pass carries no more partials than there are directions
    const int K = ndir == 1 ? 1 : precision == KS_FP64 || ndir > 4 ? 8 : ndir == 2 ? 2 : 4;
    const int nchunk = (ndir + K - 1) / K;
    // directions padded to whole chunks
    std::vector<double> hd(size_t(nchunk) * K * np, 0.0);
    if (!lnL) KS_CUDA(c, cudaMemcpy(hd.data(), dirs, size_t(ndir) * np * sizeof(double), cudaMemcpyDefault));
    for (double v : hd) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite direction");
    KS_CUDA(c, c->jvp_in.ensure((hp.size() + hd.size() + 1) * sizeof(double)));
    double* dp = c->jvp_in.as<double>();
    KS_CUDA(c, cudaMemcpyAsync(dp, hp.data(), hp.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    KS_CUDA(c, cudaMemcpyAsync(dp + np, hd.data(), hd.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    const int ncombo = nframes * nfreq;
    std::vector<double> hc(2 * size_t(ncombo));
    for (int fv = 0; fv < nfreq; ++fv)
        for (int ft = 0; ft < nframes; ++ft) {
            hc[size_t(fv) * nframes + ft] = ht[ft];
            hc[ncombo + size_t(fv) * nframes + ft] = hnu[fv];
        }
    KS_CUDA(c, c->combos.ensure(hc.size() * sizeof(double)));
    KS_CUDA(c, cudaMemcpyAsync(c->combos.p, hc.data(), hc.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    const double* dct = c->combos.as<double>();
    const double* dcn = dct + ncombo;
    const long long nrc = c->npix * ncombo;
    KS_CUDA(c, c->out_sorted.ensure(size_t(nrc) * 4 * sizeof(double)));
    KS_CUDA(c, c->jvp_out.ensure(size_t(K) * nrc * 4 * sizeof(double)));
    cudaEventRecord(c->ev0, c->stream);
    if (precision == KS_MIXED) {
        // the mixed J v reads the samples of the FP32 stream (the march once for every chunk)
        c->geo64 = geo;
        int s = launch_stream(c);
        if (s) return s;
    }
    for (int ch = 0; ch < nchunk; ++ch) {
        const double* dd = dp + np + (long long)ch * K * np;
        int s;
        const int ld = lnL ? 0 : -1;
        if (precision == KS_FP64)
            s = K == 1 ? jvp_chunk<double, 1>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld)
                       : jvp_chunk<double, 8>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld);
        else
            s = K == 1 ? jvp_chunk<float, 1>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld)
                       : K == 2 ? jvp_chunk<float, 2>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld)
                       : K == 4 ? jvp_chunk<float, 4>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld)
                                : jvp_chunk<float, 8>(c, ntot, dp, dd, np, dct, dcn, ncombo, L, nmax, slab, c->out_sorted.as<double>(), c->jvp_out.as<double>(), ld);
        if (s) return s;
        const int nd = std::min(K, ndir - ch * K);
        s = emit(c, c->jvp_out.as<double>(), 4, int(nd * ncombo), order, dimage + (long long)ch * K * nrc * 4);
        if (s) return s;
    }
    cudaEventRecord(c->ev1, c->stream);
    if (image) {
        int s = emit(c, c->out_sorted.as<double>(), 4, ncombo, order, image);
        if (s) return s;
    }
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->adjoint_ms += ms;
    return KS_OK;
}

}  // namespace

extern "C" {

int ks_jvp(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus, int32_t nfreq,
           double L, int32_t precision, int32_t nmax, double slab, const double* dirs, int32_t ndir, double* dimage, int32_t order,
           double* image) {
    return jvp_impl(c, sets, nsets, times, nframes, nus, nfreq, L, precision, nmax, slab, dirs, ndir, dimage, order, image, false);
}

int ks_spacetime_derivatives(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus,
                             int32_t nfreq, double L, int32_t precision, int32_t nmax, double slab, double* dimage, double* image) {
    if (!c || !dimage || !sets || nsets < 1) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nframes < 1 || nfreq < 1 || !times || !nus) return fail(c, KS_ERR_ARGUMENT, "need at least one frame and one frequency");
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (!(std::isfinite(L) && L > 0)) return fail(c, KS_ERR_NONFINITE, "length unit must be finite and positive");
    KS_CUDA(c, cudaSetDevice(c->device));
    std::vector<double> ht(nframes), hnu(nfreq);
    KS_CUDA(c, cudaMemcpy(ht.data(), times, nframes * sizeof(double), cudaMemcpyDefault));
    KS_CUDA(c, cudaMemcpy(hnu.data(), nus, nfreq * sizeof(double), cudaMemcpyDefault));
    for (double v : ht) if (!std::isfinite(v)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    for (double v : hnu) if (!(std::isfinite(v) && v > 0)) return fail(c, KS_ERR_NONFINITE, "frequencies must be finite and positive");
    int ntot = 0;
    {
        int s = build_tables(c, sets, nsets, &ntot, false);
        if (s) return s;
    }
    const int ncombo = nframes * nfreq;
    std::vector<double> hc(2 * size_t(ncombo));
    for (int fv = 0; fv < nfreq; ++fv)
        for (int ft = 0; ft < nframes; ++ft) {
            hc[size_t(fv) * nframes + ft] = ht[ft];
            hc[ncombo + size_t(fv) * nframes + ft] = hnu[fv];
        }
    KS_CUDA(c, c->combos.ensure(hc.size() * sizeof(double)));
    KS_CUDA(c, cudaMemcpyAsync(c->combos.p, hc.data(), hc.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    const double* dct = c->combos.as<double>();
    const long long n = c->npix;
    const long long nrc = n * ncombo;
    // the dual table, the dual anchor records, then the per-(ray, combination) value + 3 partials
    const long long ntab = (long long)ntot * ST_COUNT + c->nkv;
    const size_t tab_bytes = (size_t(std::max<long long>(ntab, 1)) * sizeof(D3) + 255) / 256 * 256;
    const size_t rec_bytes = size_t(c->total_anchors) * SA_COUNT * sizeof(D3);
    KS_CUDA(c, c->jvp_tab.ensure(tab_bytes + rec_bytes));
    D3* dtab = c->jvp_tab.as<D3>();
    D3* rec = reinterpret_cast<D3*>(static_cast<unsigned char*>(c->jvp_tab.p) + tab_bytes);
    KS_CUDA(c, c->st_buf.ensure(size_t(nrc) * 16 * sizeof(double)));
    cudaEventRecord(c->ev0, c->stream);
    if (ntab > 0) {
        k_lift_table<<<nblocks(ntab, 256), 256, 0, c->stream>>>(ntab, c->tab.as<double>(), dtab);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    const PlanView P = plan_view(c);
    k_st_anchors<<<dim3(nblocks(n, 64), c->max_nanch), 64, 0, c->stream>>>(P, c->st, n, rec);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    k_st_prefix<<<nblocks(n, 64), 64, 0, c->stream>>>(P, n, rec);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    k_spacetime_dual<<<nblocks(nrc, 64), 64, 0, c->stream>>>(P, c->st, n, rec, dtab, ntot, dct, dct + ncombo, ncombo, L, nmax, slab,
                                                             c->st_buf.as<double>());
    c->launches++;
    c->adjoint_launches++;
    KS_CUDA(c, cudaGetLastError());
    // screen order: dimage (3 x ncombo x npix x 4) and the image
    const bool dev = is_device_ptr(dimage);
    const bool idev = image && is_device_ptr(image);
    const size_t n4 = size_t(nrc) * 4;
    KS_CUDA(c, c->stage_out.ensure(n4 * 4 * sizeof(double)));
    double* dd = dev ? dimage : c->stage_out.as<double>();
    double* di = image ? (idev ? image : c->stage_out.as<double>() + 3 * n4) : nullptr;
    k_spacetime_unpack<<<nblocks(nrc, 256), 256, 0, c->stream>>>(c->st_buf.as<double>(), c->perm.as<long long>(), n, ncombo, dd, di);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    cudaEventRecord(c->ev1, c->stream);
    if (!dev) KS_CUDA(c, cudaMemcpyAsync(dimage, dd, n4 * 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (image && !idev) KS_CUDA(c, cudaMemcpyAsync(image, di, n4 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->adjoint_ms += ms;
    return KS_OK;
}

int ks_normal_matrix(ks_context* c, const double* J, int64_t m, int64_t n, int32_t precision, double* A) {
    if (!c || !J || !A || m < 1 || n < 1) return KS_ERR_ARGUMENT;
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (n > (1 << 16)) return fail(c, KS_ERR_ARGUMENT, "too many columns (%lld)", (long long)n);
    KS_CUDA(c, cudaSetDevice(c->device));
    const double* dJ = nullptr;
    {
        int s = stage_dev(c, c->dstage, J, size_t(m) * n, &dJ);
        if (s) return s;
    }
    const bool dev = is_device_ptr(A);
    double* dA = A;
    if (!dev) { KS_CUDA(c, c->stage_out.ensure(size_t(n) * n * sizeof(double))); dA = c->stage_out.as<double>(); }
    const int nb = int((n + 31) / 32);
    if (precision == KS_FP64) {
        k_normal_fp64<<<dim3(nb, nb), dim3(32, 8), 0, c->stream>>>(m, int(n), dJ, dA);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    } else {
        // 3xTF32 tensor-core GEMM: A = J^T J = Jt Jt^T from a split, transposed FP32 copy Jt[n][m]
        const long long ldj = ksdft::pad4(m);
        KS_CUDA(c, c->dft_a.ensure(size_t(n) * ldj * 2 * sizeof(float) + size_t(n) * n * sizeof(float)));
        float* jt_h = c->dft_a.as<float>();
        float* jt_l = jt_h + n * ldj;
        float* Af = jt_l + n * ldj;
        k_transpose_split<<<dim3(nb, unsigned((m + 31) / 32)), dim3(32, 8), 0, c->stream>>>(m, int(n), dJ, jt_h, jt_l, ldj);
        c->launches++;
        int s = gemm(c, int(n), int(n), int(m), jt_h, jt_l, ldj, jt_h, jt_l, ldj, Af, n);
        if (s) return s;
        k_to_f64<<<nblocks(n * n, 256), 256, 0, c->stream>>>(n * n, Af, dA);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    if (!dev) KS_CUDA(c, cudaMemcpyAsync(A, dA, size_t(n) * n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return KS_OK;
}

int ks_sample_adjoint(ks_context* c, int64_t n, const double* in, const double* Dl, const double* w, const double* R, int32_t method,
                      double* out) {
    if (!c || n < 0 || (n > 0 && (!in || !Dl || !w || !R || !out))) return KS_ERR_ARGUMENT;
    if (method != 0 && method != 1) return fail(c, KS_ERR_ARGUMENT, "method must be 0 (structured) or 1 (duals)");
    if (n == 0) return KS_OK;
    KS_CUDA(c, cudaSetDevice(c->device));
    const size_t sizes[4] = {size_t(n) * 11, size_t(n), size_t(n) * 4, size_t(n) * 4};
    const double* src[4] = {in, Dl, w, R};
    const double* dev[4];
    for (int q = 0; q < 4; ++q) {
        int s = stage_dev(c, c->dft_in[q], src[q], sizes[q], &dev[q]);
        if (s) return s;
    }
    const bool dout = is_device_ptr(out);
    double* o = out;
    if (!dout) { KS_CUDA(c, c->stage_out.ensure(size_t(n) * 31 * sizeof(double))); o = c->stage_out.as<double>(); }
    k_sample_adjoint<<<nblocks(n), kBlock, 0, c->stream>>>(n, dev[0], dev[1], dev[2], dev[3], method, o);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    if (!dout) KS_CUDA(c, cudaMemcpyAsync(out, o, size_t(n) * 31 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return KS_OK;
}

int ks_vis_chi2_gradient(ks_context* c, const ks_splat_set* sets, int32_t nsets, double t_obs, double nu, double L, int32_t precision,
                         int32_t nmax, double slab, int64_t nuv, const double* u, const double* v, const double* tap, const double* g,
                         const double* vis, const double* sigma, double psize, double scale, double* chi2, double* dparams,
                         int32_t accumulate, double* image) {
    if (!c || !u || !v || !vis || !sigma || nuv < 1) return KS_ERR_ARGUMENT;
    const VisData vd{nuv, u, v, tap, g, vis, sigma, psize, scale};
    return adjoint_run(c, sets, nsets, &t_obs, 1, &nu, 1, L, precision, nmax, slab, nullptr, KS_ORDER_SCREEN, nullptr, nullptr, 0.0,
                       nullptr, chi2, dparams, accumulate, image, &vd);
}

int ks_autotune(ks_context* c, const ks_splat_set* sets, int32_t nsets, const double* times, int32_t nframes, const double* nus,
                int32_t nfreq, double L, int32_t nmax, double slab, int32_t trials, int32_t* block, int32_t* units, double* best_ms) {
    if (!c || trials < 1) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    KS_CUDA(c, cudaSetDevice(c->device));
    const long long n4 = c->npix * (long long)nframes * nfreq * 4;
    if (nframes < 1 || nfreq < 1) return fail(c, KS_ERR_ARGUMENT, "need at least one frame and one frequency");
    KS_CUDA(c, c->st_buf.ensure(size_t(n4) * sizeof(double)));
    const int cand_nt[2] = {256, 128}, cand_u[4] = {2, 4, 8, 16};
    double best = 1e300;
    int bnt = 0, bu = 0;
    const int save_nt = c->tune_nt, save_u = c->tune_units;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 4; ++b) {
            c->tune_nt = cand_nt[a]; c->tune_units = cand_u[b];
            int s = ks_render(c, sets, nsets, times, nframes, nus, nfreq, L, KS_MIXED, nmax, slab, c->st_buf.as<double>(), KS_ORDER_SORTED);
            if (s) { c->tune_nt = save_nt; c->tune_units = save_u; return s; }
            const double before = c->kernel_ms;
            for (int t = 0; t < trials; ++t) {
                s = ks_render(c, sets, nsets, times, nframes, nus, nfreq, L, KS_MIXED, nmax, slab, c->st_buf.as<double>(), KS_ORDER_SORTED);
                if (s) { c->tune_nt = save_nt; c->tune_units = save_u; return s; }
            }
            const double ms = (c->kernel_ms - before) / trials;
            if (ms < best) { best = ms; bnt = cand_nt[a]; bu = cand_u[b]; }
        }
    c->tune_nt = bnt; c->tune_units = bu;
    if (block) *block = bnt;
    if (units) *units = bu;
    if (best_ms) *best_ms = best;
    return KS_OK;
}

int ks_adjoint_stats(ks_context* c, double* adjoint_ms, long long* launches, int reset) {
    if (!c) return KS_ERR_ARGUMENT;
    if (adjoint_ms) *adjoint_ms = c->adjoint_ms;
    if (launches) *launches = c->adjoint_launches;
    if (reset) { c->adjoint_ms = 0.0; c->adjoint_launches = 0; }
    return KS_OK;
}

}  // extern "C"

// ---- visibilities (device_visibilities.jl:53-111) ------------------------------------------------

namespace {

// Stage the DFT inputs (host or device) into device buffers; returns device pointers.
int dft_stage(ks_context* c, int slot, const double* src, size_t count, const double** dev) {
    if (!src) { *dev = nullptr; return KS_OK; }
    return stage_in(c, c->dft_in[slot], src, count * sizeof(double), reinterpret_cast<const void**>(dev));
}

int dft_checks(ks_context* c, int64_t nuv, double psize, double scale, int32_t precision) {
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first (the screen and its sort order)");
    if (nuv < 1) return fail(c, KS_ERR_ARGUMENT, "need at least one baseline");
    if (!(std::isfinite(psize) && psize > 0 && std::isfinite(scale))) return fail(c, KS_ERR_NONFINITE, "pixel size and scale must be finite");
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    return KS_OK;
}

// The twiddle tables of the separable transform: Tv[j][2k + c] (m_j, v_k, plain FP32, read by the
// combine and seed kernels) and the split GEMM operands Tu[i][2k + c] (the adjoint's B, K = 2 nuv) and
// TuT[2k + c][i] (the forward's B, K = na), both from (l_i, u_k).
struct Twiddles {
    float *tu_h, *tu_l, *tut_h, *tut_l;
    long long ldu, ldut;
};

Twiddles twiddle_layout(ks_context* c, int64_t nuv) {
    Twiddles t;
    const int na = c->nalpha;
    t.ldu = ksdft::pad4(2 * nuv);
    t.ldut = ksdft::pad4(na);
    t.tu_h = c->dft_tu.as<float>();
    t.tu_l = t.tu_h + na * t.ldu;
    t.tut_h = t.tu_l + na * t.ldu;
    t.tut_l = t.tut_h + 2 * nuv * t.ldut;
    return t;
}

int dft_twiddles(ks_context* c, int64_t nuv, const double* du, const double* dv, double psize) {
    const int na = c->nalpha, nb = c->nbeta;
    KS_CUDA(c, c->dft_tu.ensure((size_t(na) * ksdft::pad4(2 * nuv) * 2 + size_t(2 * nuv) * ksdft::pad4(na) * 2) * sizeof(float)));
    KS_CUDA(c, c->dft_tv.ensure(size_t(nb) * 2 * nuv * sizeof(float)));
    const Twiddles t = twiddle_layout(c, nuv);
    const long long nu = (long long)na * nuv;
    ksdft::k_twiddle_split<<<nblocks(nu, 256), 256, 0, c->stream>>>(na, -1.0, psize, nuv, du, 0, t.tu_h, t.tu_l, t.ldu);
    ksdft::k_twiddle_split<<<nblocks(nu, 256), 256, 0, c->stream>>>(na, -1.0, psize, nuv, du, 1, t.tut_h, t.tut_l, t.ldut);
    ksdft::k_twiddle<<<nblocks((long long)nb * nuv, 256), 256, 0, c->stream>>>(nb, 1.0, psize, nuv, dv, c->dft_tv.as<float>(), 2 * nuv);
    c->launches += 3;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// cuTensorMapEncodeTiled from the driver, through the runtime (no link against libcuda)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

// A split operand (rows x K floats, row stride ld) as 128-row x 32-float boxes with the 128-byte
// swizzle; reads past K or past the last row are zero-filled.
bool operand_map(CUtensorMap* m, const float* p, long long rows, long long K, long long ld) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(p) & 15) || (ld & 3)) return false;
    cuuint64_t dims[2] = {cuuint64_t(K), cuuint64_t(rows)};
    cuuint64_t strides[1] = {cuuint64_t(ld) * sizeof(float)};
    cuuint32_t box[2] = {cuuint32_t(ksdft::TC_BK), cuuint32_t(ksdft::TC_BM)};
    cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// C[M][N] = A[M][K] B[N][K]^T in 3xTF32 from split operands (ksdft): the tcgen05 kernel unless the
// context selects the mma.sync fallback. Outside a graph capture, the tcgen05 path reads the device
// flag after the launch, so a wait that gave up fails the call with KS_ERR_TIMEOUT.
int gemm(ks_context* c, int M, int N, int K, const float* Ah, const float* Al, long long lda, const float* Bh, const float* Bl, long long ldb,
         float* C, long long ldc) {
    if (M < 1 || N < 1) return KS_OK;
    if (K < 1) {
        KS_CUDA(c, cudaMemset2DAsync(C, size_t(ldc) * sizeof(float), 0, size_t(N) * sizeof(float), size_t(M), c->stream));
        return KS_OK;
    }
    c->launches++;
    c->kernel_launches++;
    const bool timed = !c->capturing;
    if (c->tensor_path == 1) {
        dim3 grid(unsigned((N + ksdft::BN - 1) / ksdft::BN), unsigned((M + ksdft::BM - 1) / ksdft::BM));
        if (timed) cudaEventRecord(c->evg0, c->stream);
        ksdft::k_gemm_3xtf32<<<grid, ksdft::NTHREADS, 0, c->stream>>>(M, N, K, Ah, Al, lda, Bh, Bl, ldb, C, ldc);
        KS_CUDA(c, cudaGetLastError());
    } else {
        CUtensorMap tah, tal, tbh, tbl;
        if (!operand_map(&tah, Ah, M, K, lda) || !operand_map(&tal, Al, M, K, lda) || !operand_map(&tbh, Bh, N, K, ldb) ||
            !operand_map(&tbl, Bl, N, K, ldb))
            return fail(c, KS_ERR_DEVICE, "tensor-core GEMM: cannot describe the operands as TMA tensor maps (M %d, N %d, K %d)", M, N, K);
        {
            static std::mutex mu;
            static unsigned long long done_devices = 0;   // one bit per device: the shared-memory opt-in is per device
            std::lock_guard<std::mutex> lock(mu);
            if (!(done_devices >> (c->device & 63) & 1)) {
                KS_CUDA(c, cudaFuncSetAttribute(ksdft::k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, ksdft::TC_SMEM));
                done_devices |= 1ull << (c->device & 63);
            }
        }
        // a wait gives up after ~1 s at the maximum SM clock (10 ms under the staging test hook)
        const long long limit = c->stage_test ? 20000000LL : 2000000000LL;
        dim3 grid(unsigned((N + ksdft::TC_BN - 1) / ksdft::TC_BN), unsigned((M + ksdft::TC_BM - 1) / ksdft::TC_BM));
        if (timed) cudaEventRecord(c->evg0, c->stream);
        ksdft::k_gemm_tc<<<grid, ksdft::TC_THREADS, ksdft::TC_SMEM, c->stream>>>(M, N, K, tah, tal, tbh, tbl, C, ldc, limit, c->stage_test,
                                                                              c->errflag.as<unsigned>());
        KS_CUDA(c, cudaGetLastError());
    }
    if (!timed) return KS_OK;
    cudaEventRecord(c->evg1, c->stream);
    KS_CUDA(c, cudaEventSynchronize(c->evg1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->evg0, c->evg1);
    c->gemm_ms += ms;
    c->gemm_flops += 6.0 * M * double(N) * K;
    c->gemm_launches++;
    return c->tensor_path == 1 ? KS_OK : check_device_flag(c, "tensor-core GEMM");
}

// V (nuv x 4 complex) of a device image
int dft_forward(ks_context* c, const double* dimg, int32_t order, int64_t nuv, const double* du, const double* dv, const double* dtap,
                double psize, double scale, int32_t precision, double* dV) {
    const int na = c->nalpha, nb = c->nbeta;
    const long long* inv = order == KS_ORDER_SORTED ? c->inv_perm.as<long long>() : nullptr;
    if (precision == KS_FP64) {
        ksdft::k_vis_direct<<<nblocks(nuv, 64), 64, 0, c->stream>>>(na, nb, dimg, inv, nuv, du, dv, dtap, psize, scale, dV);
        c->launches++;
        c->kernel_launches++;
        KS_CUDA(c, cudaGetLastError());
        return KS_OK;
    }
    int s = dft_twiddles(c, nuv, du, dv, psize);
    if (s) return s;
    const Twiddles t = twiddle_layout(c, nuv);
    const long long lda = ksdft::pad4(na), ldt = ksdft::pad4(2 * nuv);
    KS_CUDA(c, c->dft_a.ensure(size_t(2) * 4 * nb * lda * sizeof(float)));
    KS_CUDA(c, c->dft_t.ensure(size_t(4) * nb * ldt * sizeof(float)));
    float* a_h = c->dft_a.as<float>();
    float* a_l = a_h + 4LL * nb * lda;
    ksdft::k_pack_image<<<nblocks((long long)na * nb, 256), 256, 0, c->stream>>>(dimg, inv, na, nb, a_h, a_l, lda);
    c->launches++;
    if ((s = gemm(c, 4 * nb, int(2 * nuv), na, a_h, a_l, lda, t.tut_h, t.tut_l, t.ldut, c->dft_t.as<float>(), ldt))) return s;
    ksdft::k_vis_combine<<<dim3(unsigned((nuv + ksdft::VC_K - 1) / ksdft::VC_K), 4), ksdft::VC_K * ksdft::VC_G, 0, c->stream>>>(
        nb, nuv, c->dft_t.as<float>(), ldt, c->dft_tv.as<float>(), 2 * nuv, dtap, scale, dV);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// seed (npix x 4) of device weights w (nuv x 4 complex)
int dft_adjoint(ks_context* c, const double* dw, int64_t nuv, const double* du, const double* dv, const double* dtap, double psize,
                double scale, int32_t precision, double* dseed, int32_t order, bool have_twiddles) {
    const int na = c->nalpha, nb = c->nbeta;
    const long long* inv = order == KS_ORDER_SORTED ? c->inv_perm.as<long long>() : nullptr;
    if (precision == KS_FP64) {
        ksdft::k_seed_direct<<<nblocks((long long)na * nb, 64), 64, 0, c->stream>>>(na, nb, inv, nuv, dw, du, dv, dtap, psize, scale, dseed);
        c->launches++;
        c->kernel_launches++;
        KS_CUDA(c, cudaGetLastError());
        return KS_OK;
    }
    if (!have_twiddles) {
        int s = dft_twiddles(c, nuv, du, dv, psize);
        if (s) return s;
    }
    const Twiddles t = twiddle_layout(c, nuv);
    const long long ldc = ksdft::pad4(2 * nuv);
    KS_CUDA(c, c->dft_c.ensure(size_t(2) * 4 * nb * ldc * sizeof(float)));
    const long long lds = ksdft::pad4(na);
    KS_CUDA(c, c->dft_s.ensure(size_t(4) * nb * lds * sizeof(float)));
    float* c_h = c->dft_c.as<float>();
    float* c_l = c_h + 4LL * nb * ldc;
    ksdft::k_seed_rhs<<<nblocks(nuv * 4 * nb, 256), 256, 0, c->stream>>>(nb, nuv, c->dft_tv.as<float>(), 2 * nuv, dw, dtap, scale, c_h, c_l, ldc);
    c->launches++;
    // S[(s, j)][i] = CT Tu^T: rows of the seed image, so that the unpacking reads along i
    int s = gemm(c, 4 * nb, na, int(2 * nuv), c_h, c_l, ldc, t.tu_h, t.tu_l, t.ldu, c->dft_s.as<float>(), lds);
    if (s) return s;
    ksdft::k_unpack_seed<<<nblocks((long long)na * nb, 256), 256, 0, c->stream>>>(c->dft_s.as<float>(), lds, na, nb, inv, dseed);
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// copy `count` doubles from the device buffer `src` to `dst` (host or device)
int deliver(ks_context* c, const double* src, double* dst, size_t count) {
    KS_CUDA(c, cudaMemcpyAsync(dst, src, count * sizeof(double), cudaMemcpyDefault, c->stream));
    return KS_OK;
}

}  // namespace

extern "C" {

int ks_visibilities(ks_context* c, const double* image, int32_t order, int64_t nuv, const double* u, const double* v, const double* tap,
                    double psize, double scale, int32_t precision, double* V) {
    if (!c || !image || !u || !v || !V) return KS_ERR_ARGUMENT;
    int s = dft_checks(c, nuv, psize, scale, precision);
    if (s) return s;
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    KS_CUDA(c, cudaSetDevice(c->device));
    const double *dimg, *du, *dv, *dtap;
    if ((s = dft_stage(c, 0, image, size_t(c->npix) * 4, &dimg)) || (s = dft_stage(c, 1, u, nuv, &du)) || (s = dft_stage(c, 2, v, nuv, &dv)) ||
        (s = dft_stage(c, 3, tap, tap ? nuv : 0, &dtap)))
        return s;
    KS_CUDA(c, c->dft_in[4].ensure(size_t(nuv) * 8 * sizeof(double)));
    cudaEventRecord(c->ev0, c->stream);
    if ((s = dft_forward(c, dimg, order, nuv, du, dv, dtap, psize, scale, precision, c->dft_in[4].as<double>()))) return s;
    cudaEventRecord(c->ev1, c->stream);
    if ((s = deliver(c, c->dft_in[4].as<double>(), V, size_t(nuv) * 8))) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c->ev0, c->ev1);
    c->kernel_ms += ms;
    return KS_OK;
}

int ks_vis_seed(ks_context* c, const double* w, int64_t nuv, const double* u, const double* v, const double* tap, double psize, double scale,
                int32_t precision, double* seed, int32_t order) {
    if (!c || !w || !u || !v || !seed) return KS_ERR_ARGUMENT;
    int s = dft_checks(c, nuv, psize, scale, precision);
    if (s) return s;
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    KS_CUDA(c, cudaSetDevice(c->device));
    const double *dw, *du, *dv, *dtap;
    if ((s = dft_stage(c, 0, w, size_t(nuv) * 8, &dw)) || (s = dft_stage(c, 1, u, nuv, &du)) || (s = dft_stage(c, 2, v, nuv, &dv)) ||
        (s = dft_stage(c, 3, tap, tap ? nuv : 0, &dtap)))
        return s;
    KS_CUDA(c, c->dft_in[5].ensure(size_t(c->npix) * 4 * sizeof(double)));
    if ((s = dft_adjoint(c, dw, nuv, du, dv, dtap, psize, scale, precision, c->dft_in[5].as<double>(), order, false))) return s;
    if ((s = deliver(c, c->dft_in[5].as<double>(), seed, size_t(c->npix) * 4))) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return KS_OK;
}

int ks_frame_chi2_seed(ks_context* c, const double* image, int32_t order, int64_t nuv, const double* u, const double* v, const double* tap,
                       const double* g, const double* vis, const double* sigma, double psize, double scale, int32_t precision,
                       double* chi2, double* seed) {
    if (!c || !image || !u || !v || !vis || !sigma || !chi2 || !seed) return KS_ERR_ARGUMENT;
    int s = dft_checks(c, nuv, psize, scale, precision);
    if (s) return s;
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    KS_CUDA(c, cudaSetDevice(c->device));
    const double *dimg, *du, *dv, *dtap, *dg, *dvis, *dsig;
    if ((s = dft_stage(c, 0, image, size_t(c->npix) * 4, &dimg)) || (s = dft_stage(c, 1, u, nuv, &du)) || (s = dft_stage(c, 2, v, nuv, &dv)) ||
        (s = dft_stage(c, 3, tap, tap ? nuv : 0, &dtap)) || (s = dft_stage(c, 6, g, g ? 2 * nuv : 0, &dg)) ||
        (s = dft_stage(c, 7, vis, size_t(nuv) * 8, &dvis)))
        return s;
    KS_CUDA(c, c->dft_in[4].ensure(size_t(nuv) * 8 * sizeof(double) * 2 + size_t(nuv) * 4 * sizeof(double)));
    double* dV = c->dft_in[4].as<double>();
    double* dW = dV + nuv * 8;
    double* dS = dW + nuv * 8;
    KS_CUDA(c, cudaMemcpyAsync(dS, sigma, size_t(nuv) * 4 * sizeof(double), cudaMemcpyDefault, c->stream));
    dsig = dS;
    KS_CUDA(c, c->dft_in[5].ensure(size_t(c->npix) * 4 * sizeof(double)));
    if ((s = dft_forward(c, dimg, order, nuv, du, dv, dtap, psize, scale, precision, dV))) return s;
    const int nblk = int((nuv * 4 + 255) / 256);
    KS_CUDA(c, c->dft_partial.ensure(size_t(nblk) * sizeof(double)));
    ksdft::k_chi2_weights<<<nblk, 256, 0, c->stream>>>(nuv, dV, dg, dvis, dsig, dW, c->dft_partial.as<double>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    if ((s = dft_adjoint(c, dW, nuv, du, dv, dtap, psize, scale, precision, c->dft_in[5].as<double>(), order, precision != KS_FP64))) return s;
    std::vector<double> part(nblk);
    KS_CUDA(c, cudaMemcpyAsync(part.data(), c->dft_partial.p, nblk * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if ((s = deliver(c, c->dft_in[5].as<double>(), seed, size_t(c->npix) * 4))) return s;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    double x = 0.0;
    for (double p : part) x += p;   // fixed order: deterministic
    *chi2 = x;
    return KS_OK;
}

}  // extern "C"

// ---- the allocation-free thin image -------------------------------------------------------------

// Device address of g_noalloc_tab, looked up once per device (with that device current) by the first
// ks_thin_image_noalloc call on it. cudaGetSymbolAddress does not allocate.
static std::mutex g_noalloc_mutex;
static void* g_noalloc_addr[64] = {nullptr};

static int noalloc_table(ks_context* c, double** tab) {
    if (c->device < 0 || c->device >= 64) return fail(c, KS_ERR_DEVICE, "device index %d out of range", c->device);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[c->device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_tab);
        if (e != cudaSuccess || !p) return cuda_fail(c, e == cudaSuccess ? cudaErrorInvalidSymbol : e, "cudaGetSymbolAddress(g_noalloc_tab)");
        g_noalloc_addr[c->device] = p;
    }
    *tab = static_cast<double*>(g_noalloc_addr[c->device]);
    return KS_OK;
}

extern "C" {

int ks_thin_image_noalloc(ks_context* c, const double* params, int32_t nsplat, double t_obs, int32_t precision, double* out,
                          int32_t order) {
    if (!c) return KS_ERR_ARGUMENT;
    if (!c->regenerated) return fail(c, KS_ERR_NOT_REGENERATED, "regenerate the context first");
    if (nsplat < 0 || nsplat > kNoAllocMaxSplats)
        return fail(c, KS_ERR_ARGUMENT, "ks_thin_image_noalloc takes at most %d splats (got %d)", kNoAllocMaxSplats, nsplat);
    if (precision != KS_FP64 && precision != KS_MIXED) return fail(c, KS_ERR_ARGUMENT, "unknown precision %d", precision);
    if (order != KS_ORDER_SORTED && order != KS_ORDER_SCREEN) return fail(c, KS_ERR_ARGUMENT, "unknown order %d", order);
    if (!std::isfinite(t_obs)) return fail(c, KS_ERR_NONFINITE, "non-finite observation time");
    KS_CUDA(c, cudaSetDevice(c->device));
    if (!is_device_ptr(out) || (nsplat > 0 && !is_device_ptr(params)))
        return fail(c, KS_ERR_ARGUMENT, "ks_thin_image_noalloc needs device pointers for params and out");
    double* tab = nullptr;
    int s = noalloc_table(c, &tab);
    if (s) return s;
    const long long n = c->npix;
    if (nsplat > 0) {
        SetDesc d{KS_THIN14, 14, nsplat, 0, params, nullptr, 0.0};
        k_splat_table<<<nblocks(nsplat, 64), 64, 0, c->stream>>>(d, tab);
        c->launches++;
        KS_CUDA(c, cudaGetLastError());
    }
    const long long* perm = order == KS_ORDER_SCREEN ? c->perm.as<long long>() : nullptr;
    int sl = precision == KS_FP64 ? launch_thin<double>(c, tab, nsplat, t_obs, perm, out, false) : launch_thin<float>(c, tab, nsplat, t_obs, perm, out, false);
    if (sl) return sl;
    KS_CUDA(c, cudaStreamSynchronize(c->stream));
    return KS_OK;
}

}  // extern "C"
