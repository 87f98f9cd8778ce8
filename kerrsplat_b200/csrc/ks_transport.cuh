// ks_transport.cuh -- the polarized transport over a sample stream: every frame and frequency of a render,
// in FP32 (the mixed path) or FP64 (the plain path).
//
// A block's work unit is 32 neighbouring rays (sorted slots) x one segment of their samples x one frame x up
// to CH frequencies. It takes the segment in runs of R samples, front to back. What the reference does per
// sample (transport.jl:190-198: every element's coefficients, their sum, one exact step, compositing) is
// done for a whole run at a time, phase by phase:
//   1. tests: every (ray, sample) against the run's candidate splats (support and weight cutoff), the passing
//      splats as bit masks in shared memory;
//   2. evaluation: the samples with a passing splat, dealt to the threads in the order of their number of
//      splats, so that the lanes of a warp do the same amount of work. A thread forms its sample's frame once,
//      sums its splats' coefficients at every frequency in splat order in registers, and leaves them
//      in its record; then the exact step of every (frequency, sample) takes their place: the four scalars of
//      O = sum o_n K^n, the six entries of K, and E;
//   3. composition: one thread per (ray, row of P, frequency) takes the ray's records front to back
//      (s += p E, p <- p O, step.jl:347) as three products with the sparse K each.
// The sums of a sample do not depend on the order in which samples are dealt, so the image is the same bit
// for bit from call to call.
//
// Bound by instruction issue (coefficient fits and steps). The block-cooperative consumer before it took one
// sample at a time, with some eight block barriers for each: 17.1 ms at 256 x 256 x 1024, 64 splats,
// three frequencies.
#pragma once
#include "ks_gradient.cuh"
#include "ks_mixed.cuh"

namespace ks {

// ---- splat rows ------------------------------------------------------------------------------------------
// What the transport reads of a splat, in the order of use, with everything that depends on the splat alone
// formed in FP64: A = R diag(exp(-s)) (the whitened rotation), the velocity's gamma and 1 / (gamma + 1), the
// cyclotron frequency, the centre's angle at t0. A row is an odd number of 16-byte words, so that lanes on
// different splats read different banks.
enum RowField {
    RW_CX, RW_CY, RW_CZ, RW_T0, RW_OMEGA, RW_INVW, RW_NE, RW_RHO,
    RW_A0, RW_A1, RW_A2, RW_A3, RW_A4, RW_A5, RW_A6, RW_A7, RW_A8, RW_U1, RW_U2, RW_U3,
    RW_BX, RW_BY, RW_BZ, RW_GQ, RW_GAM, RW_TE, RW_F0, RW_KR, RW_NUC, RW_SUPP, RW_KIND, RW_ANG,
    RW_THERMAL_COUNT,
    RW_DF0 = RW_THERMAL_COUNT, RW_DKR,   // thermal tables with a gradient: the Bessel ratios' derivatives by ln Te
    // scenes of several populations: the knot record, then the constants of the power-law and kappa fits
    // (population_constants)
    RW_KOFF = RW_THERMAL_COUNT, RW_NK, RW_E, RW_ECOUNT = 32, RW_COUNT = RW_E + RW_ECOUNT
};
template <class T, int KM>
__host__ __device__ constexpr int row_stride() {
    return KM == 1 ? (sizeof(T) == 4 ? 36 : 34) : (sizeof(T) == 4 ? 68 : 66);
}
static_assert(RW_DKR < 34 && RW_COUNT <= 66, "rows hold their fields");

constexpr double kNUC = kEE / (2.0 * 3.141592653589793 * kME * kCL);   // cyclotron frequency per gauss

// the logarithm of the base that hlog2 and hexp2 pair on: 2 in FP32, e in FP64
template <class T> __device__ __forceinline__ double row_log(double v) { return sizeof(T) == 4 ? log2(v) : log(v); }

// What the power-law fits (powerlaw_cs) and the kappa fits (kappa_cs) take from the splat alone, formed once in FP64:
// some twenty powers an evaluation otherwise. 112 x 112 rays x up to 2048 samples, 96 splats of three populations, four
// frequencies, two frames: k_transport 17.0 -> 12.1 ms. The wider rows (68 words against 44 in FP32) stay in global
// memory for tables that shared memory does not hold.
enum PowerField { EP_J, EP_JQ, EP_JV, EP_A, EP_AQ, EP_AV, EP_RQ, EP_RV, EP_P1, EP_PH, EP_PG };
enum KappaField {
    EK_X,                                                    // 1 / (w kappa)^2
    EK_I = 1, EK_Q = 5, EK_AI = 9, EK_AQ = 13,               // a bridge each: low limit, x slope, x ln(low / high), 1 / x
    EK_V = 17, EK_AV = 22,                                   // low, slope, ln(low / high), x, 1 / x without the pitch angle's part
    EK_FIT = 27, EK_FQ0, EK_FQ1, EK_FV0, EK_FV1 = 31         // rotativity fits: the lower one's index, the four amplitudes
};
template <class T>
__device__ void population_constants(const double* p, T* e) {
    constexpr double PI = 3.141592653589793;
    const double ej = kEE * kEE / kCL, ea = kEE * kEE / (kME * kCL);
    if (int(p[ST_KIND]) == KS_POWERLAW22) {
        const double q = p[ST_P], gm = p[ST_GMIN], sp = p[ST_GSPAN];
        e[EP_J] = T(ej * pow(3.0, q / 2) * (q - 1) / (2 * (q + 1) * sp) * p[ST_GAMJ]);
        e[EP_JQ] = T((q + 1) / (q + 7.0 / 3));
        e[EP_JV] = T(171.0 / 250 * pow(q, 49.0 / 100) * sqrt(3.0));
        e[EP_A] = T(ea * pow(3.0, (q + 1) / 2) * (q - 1) / (4 * sp) * p[ST_GAMA]);
        e[EP_AQ] = T(pow(17.0 / 500 * q - 43.0 / 1250, 43.0 / 500));
        e[EP_AV] = T(pow(71.0 / 100 * q + 22.0 / 625, 197.0 / 500));
        e[EP_RQ] = T(-ea * (q - 1) / sp * pow(gm, 2 - q) / (q / 2 - 1));
        e[EP_RV] = T(2 * (q + 2) / (q + 1) * ea * (q - 1) / sp * pow(gm, -(q + 1)) * log(gm));
        e[EP_P1] = T((q - 1) / 2);
        e[EP_PH] = T(q / 2 - 1);
        e[EP_PG] = T((q / 2 - 1) * row_log<T>(gm * gm));
    } else if (int(p[ST_KIND]) == KS_KAPPA22) {
        const double k = p[ST_KAP], w = p[ST_W], sj = (3 * k - 4) / 6, sa = (3 * k - 1) / 6;
        auto bridge = [&](int f, double scale, double lo, double hi, double xx, double slope) {
            e[f] = T(scale * lo); e[f + 1] = T(xx * slope); e[f + 2] = T(xx * row_log<T>(lo / hi)); e[f + 3] = T(1 / xx);
        };
        auto bridge_v = [&](int f, double scale, double lo, double hi, double xx, double slope) {
            e[f] = T(scale * lo); e[f + 1] = T(slope); e[f + 2] = T(row_log<T>(lo / hi)); e[f + 3] = T(xx); e[f + 4] = T(1 / xx);
        };
        e[EK_X] = T(1 / ((w * k) * (w * k)));
        const double g = 4 * PI * p[ST_G43] / (12.980246132766677 * p[ST_G2]), hk = 0.25 * pow(3.0, (k - 1) / 2) * (k - 2) * (k - 1) * p[ST_GQ] * p[ST_GP];
        bridge(EK_I, ej, g, hk, 3 * pow(k, -1.5), sj);
        bridge(EK_Q, ej, 0.5 * g, (0.64 + k / 50) * hk, 3.7 * pow(k, -1.6), sj);
        bridge_v(EK_V, ej, 0.5625 * pow(k, -66.0 / 125) / w * g, 0.765625 * pow(k, -11.0 / 25) / w * hk, 3 * pow(k, -1.5), sj);
        const double ck = (k - 2) * (k - 1) * k;
        const double base = 1.2009369551760027 * (10.0 / 41) * 4 * PI * PI / pow(w * k, 16.0 / 3 - k) * ck / (3 * k - 1) * 0.9027452929509336 * p[ST_HYP];
        const double hi = 2 * pow(PI, 2.5) / 3 * ck / pow(w * k, 5.0) * (2 * p[ST_GK2] / (2 + k) - 1);
        const double es = kEE * kNUC;   // n_e e / (B sin theta_B) = n_e es / (nu_c sin theta_B)
        bridge(EK_AI, es, base, hi * (pow(3 / k, 19.0 / 4) + 3.0 / 5), pow(-7.0 / 4 + 8 * k / 5, -43.0 / 50), sa);
        bridge(EK_AQ, es, 25.0 / 48 * base, (441 * pow(k, -144.0 / 25) + 11.0 / 20) * hi, 1.4 * pow(k, -23.0 / 20), sa);
        bridge_v(EK_AV, es, 77 / (100 * w) * pow(k, -0.7) * base,
                 14.3 * pow(w, -116.0 / 125) * (169 * pow(k, -8.0) + 13.0 / 2500 * k - 263.0 / 5000 + 47 / (200 * k)) * hi,
                 1.22 * pow(k, -142.0 / 125) + 7.0 / 1000, sa);
        const double kc = fmin(5.0, fmax(3.5, k)), s = sqrt(w), x = s * exp(-5 * w);
        const int i = kc < 4.0 ? 0 : kc < 4.5 ? 1 : 2;
        const double f = (kc - 3.5 - 0.5 * i) * 2;
        const double q[4] = {17 * w - 3 * s + 7 * x, 46 * w / 3 - 5 * s / 3 + 17 * x / 3, 14 * w - 13 * s / 8 + 9 * x / 2, 25 * w / 2 - s + 5 * x};
        const double v[4] = {(w * w + 2 * w + 1) / (25 * w * w / 8 + 4 * w + 1), (w * w + 54 * w + 50) / (30 * w * w / 11 + 134 * w + 50),
                             (w * w + 43 * w + 38) / (7 * w * w / 3 + 185 * w / 2 + 38), (w + 13.0 / 14) / (2 * w + 13.0 / 14)};
        e[EK_FIT] = T(i);
        e[EK_FQ0] = T(-ea * (1 - f) * q[i]); e[EK_FQ1] = T(-ea * f * q[i + 1]);
        e[EK_FV0] = T(2 * ea * p[ST_KB] * (1 - f) * v[i]); e[EK_FV1] = T(2 * ea * p[ST_KB] * f * v[i + 1]);
    }
}

// rows of the concatenated FP64 table, then the knot array; `total` values, the tail zero
template <class T, int KM>
__global__ void k_rows(int ntot, int nkv, long long total, const double* __restrict__ tab, const double* __restrict__ gtab, T* __restrict__ out) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    constexpr int ST = row_stride<T, KM>();
    const long long nr = (long long)ntot * ST;
    if (q >= total) return;
    if (q >= nr) { out[q] = q - nr < nkv ? T(tab[(long long)ntot * ST_COUNT + (q - nr)]) : T(0); return; }
    const double* p = tab + (q / ST) * ST_COUNT;
    const int f = int(q % ST);
    const double gam = sqrt(1.0 + p[ST_U1] * p[ST_U1] + p[ST_U2] * p[ST_U2] + p[ST_U3] * p[ST_U3]);
    double v = 0.0;
    switch (f) {
        case RW_CX: v = p[ST_CX]; break;
        case RW_CY: v = p[ST_CY]; break;
        case RW_CZ: v = p[ST_CZ]; break;
        case RW_T0: v = p[ST_T0]; break;
        case RW_OMEGA: v = p[ST_OMEGA]; break;
        case RW_INVW: v = p[ST_INVW]; break;
        case RW_NE: v = p[ST_NE]; break;
        case RW_RHO: v = p[ST_RHO]; break;
        case RW_U1: v = p[ST_U1]; break;
        case RW_U2: v = p[ST_U2]; break;
        case RW_U3: v = p[ST_U3]; break;
        case RW_BX: v = p[ST_BHX]; break;
        case RW_BY: v = p[ST_BHY]; break;
        case RW_BZ: v = p[ST_BHZ]; break;
        case RW_GQ: v = 1.0 / (gam + 1.0); break;
        case RW_GAM: v = gam; break;
        case RW_TE: v = p[ST_TE]; break;
        case RW_F0: v = p[ST_F0]; break;
        case RW_KR: v = p[ST_KR]; break;
        case RW_NUC: v = kNUC * p[ST_BMAG]; break;
        case RW_SUPP: v = p[ST_SUPP]; break;
        case RW_KIND: v = p[ST_KIND]; break;
        case RW_ANG: v = atan2(p[ST_CY], p[ST_CX]); break;
        default: break;
    }
    if (f >= RW_A0 && f <= RW_A8) v = p[ST_R0 + (f - RW_A0)] * p[ST_ES1 + (f - RW_A0) % 3];
    if (KM == 1 && gtab && f == RW_DF0) v = gtab[(q / ST) * GT_COUNT + GT_DF0];
    if (KM == 1 && gtab && f == RW_DKR) v = gtab[(q / ST) * GT_COUNT + GT_DKR];
    if (KM != 1) {
        if (f == RW_KOFF) v = p[ST_KOFF];
        else if (f == RW_NK) v = p[ST_NK];
        else if (f == RW_E) {   // one thread forms a splat's population constants
            for (int k = 0; k < RW_ECOUNT; ++k) out[q + k] = T(0);
            population_constants(p, out + q);
            return;
        } else if (f > RW_E && f < RW_COUNT) return;
    }
    out[q] = T(v);
}
static_assert(EK_FV1 < RW_ECOUNT, "rows hold the kappa constants");

// ---- hardware functions -----------------------------------------------------------------------------------
// The FP32 forms are one instruction each: the approximations that -prec-div=false and the __-functions compile
// to, with subnormal arguments and results taken as zero (the library forms rescale them, three to four
// instructions a call and some eighty a coefficient evaluation). FP64: the library's.
__device__ __forceinline__ float hrcp(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float hsqrt(float x) { float y; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float hrsqrt(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float hlog2(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float hexp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ double hrcp(double x) { return 1.0 / x; }
__device__ __forceinline__ double hsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double hrsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ double hlog2(double x) { return log(x); }    // a natural pair: only hexp2(c hlog2(x)) = x^c is formed
__device__ __forceinline__ double hexp2(double x) { return exp(x); }
// exp(x), ln(x)
__device__ __forceinline__ float hexp(float x) { return hexp2(x * 1.4426950408889634f); }
__device__ __forceinline__ float hln(float x) { return hlog2(x) * 0.6931471805599453f; }
__device__ __forceinline__ double hexp(double x) { return exp(x); }
__device__ __forceinline__ double hln(double x) { return log(x); }

// ---- the pair arithmetic ---------------------------------------------------------------------------------

// Sine and cosine of the product a b, to FP32's rounding: the product's own rounding error is carried, the reduction
// by pi/2 is in two parts (Cody & Waite 1980) and the series run on [-pi/4, pi/4]. The hardware pair is good to 4e-7,
// which moves a centre at 10 M by 4e-6 M and the weight of a splat 0.3 M wide by some 1e-5: the largest error of an
// evaluation. A test needs no better than that (its cutoff is a weight of 1e-6).
__device__ __forceinline__ void sincos_product(float a, float b, float& s, float& c) {
    const float p = a * b, lo = fmaf(a, b, -p);
    const float k = rintf(p * 0.63661977236758134f);
    float x = fmaf(-k, 1.57079637050628662f, p);
    x += fmaf(-k, -4.37113900018624283e-8f, lo);
    const float x2 = x * x;
    const float sn = fmaf(x * x2, fmaf(x2, fmaf(x2, fmaf(x2, 1.f / 362880.f, -1.f / 5040.f), 1.f / 120.f), -1.f / 6.f), x);
    const float cs = fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 1.f / 40320.f, -1.f / 720.f), 1.f / 24.f), -0.5f), 1.f);
    const int q = int(k);
    s = (q & 1) ? cs : sn;
    c = (q & 1) ? sn : cs;
    if (q & 2) s = -s;
    if ((q + 1) & 2) c = -c;
}
__device__ __forceinline__ void sincos_product(double a, double b, double& s, double& c) { fsincos(a * b, s, c); }
// exp(-q), the rounding of q log2(e) carried
__device__ __forceinline__ float weight_of(float q) {
    const float y = q * -1.4426950408889634f, lo = fmaf(q, -1.4426950408889634f, -y) - q * 1.9259629e-8f;
    const float e = hexp2(y);
    return fmaf(e, lo * 0.6931471805599453f, e);
}
__device__ __forceinline__ double weight_of(double q) { return exp(-q); }

// The weight exponent of a splat row at (t, x, y, z). TEST: as a test needs it, with splat_exponent's cull.
template <bool TEST, class T>
__device__ __forceinline__ bool row_exponent(const T* r, T t, T x, T y, T z, T& q) {
    const T dt = t - r[RW_T0];
    T sp, cp;
    if constexpr (TEST) fsincos(r[RW_OMEGA] * dt, sp, cp);
    else sincos_product(r[RW_OMEGA], dt, sp, cp);
    const T cx = r[RW_CX] * cp - r[RW_CY] * sp, cy = r[RW_CX] * sp + r[RW_CY] * cp;
    const T d0 = x - cx, d1 = y - cy, d2 = z - r[RW_CZ];
    if (TEST && d0 * d0 + d1 * d1 + d2 * d2 > r[RW_SUPP]) return false;
    const T a = d0 * cp + d1 * sp, b = -d0 * sp + d1 * cp;
    const T e0 = r[RW_A0] * a + r[RW_A3] * b + r[RW_A6] * d2;
    const T e1 = r[RW_A1] * a + r[RW_A4] * b + r[RW_A7] * d2;
    const T e2 = r[RW_A2] * a + r[RW_A5] * b + r[RW_A8] * d2;
    const T tt = dt * r[RW_INVW];
    q = (e0 * e0 + e1 * e1 + e2 * e2 + tt * tt) / T(2);
    return true;
}
template <class T>
__device__ __forceinline__ void row_knot_exponent(const T* r, const T* knots, T t, T x, T y, T z, T& q) {
    T cx, cy, cz;
    knot_centre(knots + int(r[RW_KOFF]), int(r[RW_NK]), t, cx, cy, cz);
    const T d0 = x - cx, d1 = y - cy, d2 = z - cz;
    const T e0 = r[RW_A0] * d0 + r[RW_A3] * d1 + r[RW_A6] * d2;
    const T e1 = r[RW_A1] * d0 + r[RW_A4] * d1 + r[RW_A7] * d2;
    const T e2 = r[RW_A2] * d0 + r[RW_A5] * d1 + r[RW_A8] * d2;
    const T tt = (t - r[RW_T0]) * r[RW_INVW];
    q = (e0 * e0 + e1 * e1 + e2 * e2 + tt * tt) / T(2);
}

// local_frame (frames.jl:108-128) of a splat row: 1 / g (in the field g), cos theta_B and the rotation by 2 chi straight from the
// Walker-Penrose components (cos 2chi = (x^2 - y^2) / (x^2 + y^2), sin 2chi = 2 x y / (x^2 + y^2)).
template <class T>
__device__ __forceinline__ LFrame<T> row_frame(const SampleFrame<T>& F, const T* r, T alpha, T beta, T a_sin_tho) {
    const T u1 = r[RW_U1], u2 = r[RW_U2], u3 = r[RW_U3], q = r[RW_GQ], gam = r[RW_GAM];
    const T bx = r[RW_BX], by = r[RW_BY], bz = r[RW_BZ];
    const T ud = u1 * F.pz[1] + u2 * F.pz[2] + u3 * F.pz[3];
    const T ig = gam * F.pz[0] - ud, g = hrcp(ig);
    const T udq = ud * q - F.pz[0];
    const T k0 = (F.pz[1] + u1 * udq) * g, k1 = (F.pz[2] + u2 * udq) * g, k2 = (F.pz[3] + u3 * udq) * g;
    const T cosB = k0 * bx + k1 * by + k2 * bz;
    T f0 = k1 * bz - k2 * by, f1 = k2 * bx - k0 * bz, f2 = k0 * by - k1 * bx;
    const T fn2 = f0 * f0 + f1 * f1 + f2 * f2;
    if (!(fn2 > T(0))) return {ig, cosB, T(0), T(0), T(1)};
    const T fi = hrsqrt(fn2);
    f0 *= fi; f1 *= fi; f2 *= fi;
    const T fd = u1 * f0 + u2 * f1 + u3 * f2, fdq = fd * q;
    const T fz1 = f0 + u1 * fdq, fz2 = f1 + u2 * fdq, fz3 = f2 + u3 * fdq;
    const T ft = F.lapse_inv * fd, fr = F.sDS * fz1, fth = F.misS * fz3, fph = F.om_lapse * fd + F.ivarpi * fz2;
    const T a = F.a, rr = F.r, sth = F.sth, cth = F.cth;
    const T Aw = F.pu[0] * fr - F.pu[1] * ft + a * sth * sth * (F.pu[1] * fph - F.pu[3] * fr);
    const T Bw = ((rr * rr + a * a) * (F.pu[3] * fth - F.pu[2] * fph) - a * (F.pu[0] * fth - F.pu[2] * ft)) * sth;
    const T kk1 = Aw * rr - Bw * a * cth, kk2 = -(Aw * a * cth + Bw * rr);
    const T mu = -(alpha + a_sin_tho);
    const T y = mu * kk1 - beta * kk2, x = beta * kk1 + mu * kk2;
    const T r2 = x * x + y * y;
    if (!(r2 > T(0))) return {ig, cosB, T(0), T(0), T(1)};
    const T ir = hrcp(r2);
    return {ig, cosB, T(0), T(2) * x * y * ir, (x * x - y * y) * ir};
}

// The smallest normal number: below it the hardware reciprocal is infinite.
template <class T> __device__ __forceinline__ constexpr T smallest() { return sizeof(T) == 4 ? T(1.17549435e-38) : T(2.2250738585072014e-308); }

// cap_factor (coefficients.jl:264-288) from the ratios of Q and V to I
template <class T>
__device__ __forceinline__ T ratio_cap(T q, T v) {
    const T p2 = q * q + v * v;
    return p2 > T(0.9801) ? T(0.99) * hrsqrt(p2) : T(1);
}
// ... from the coefficients; those below the smallest normal number scaled by a power of two into range
template <class T>
__device__ __forceinline__ T row_cap(T I, T Q, T V) {
    if (!(I > T(0))) return (Q == T(0) && V == T(0)) ? T(1) : T(0);
    if (!(I >= smallest<T>())) {
        const T b = sizeof(T) == 4 ? T(18446744073709551616.0) : T(1.3407807929942597e154);   // 2^64, 2^512
        I *= b; Q *= b; V *= b;
    }
    const T i = hrcp(I);
    return ratio_cap(Q * i, V * i);
}

// 1 / B_nu from exp(h nu / k T) - 1; zero where that, or its product with what follows, would overflow: a splat far too
// cold to emit, whose absorptivity is 0 / 0
template <class T>
__device__ __forceinline__ T planck_inverse(T k, T nu, T em1) {
    const T nh = nu * T(1e-11), bn = k * nh * nh * nh, i = em1 * hrcp(bn);
    return bn > T(0) && i < (sizeof(T) == 4 ? T(1e30) : T(1e300)) ? i : T(0);
}

// The thermal fits (thermal_cs, coefficients.jl:101-145): the powers of x and of nu / nu_s from one logarithm
// each, the constants folded in FP64, and one cap for the emissivities and the absorptivities (Kirchhoff's law
// gives both the same ratios). Returns false where nothing emits, absorbs or rotates.
template <class T>
__device__ __forceinline__ bool thermal_row(const T* r, T ne, T nu, T st, T ct, T c[8]) {
    const T Te = r[RW_TE], nc = r[RW_NUC], f0 = r[RW_F0];
    const T inu = hrcp(nu), b = nc * inu;                       // nu_c / nu
    constexpr double kWP = kEE * kEE / (3.141592653589793 * kME), kRV = 3.141592653589793 * 2.0 / kCL;
    const T pl = T(kWP) * ne * inu * inu;                       // (omega_p / omega)^2
    if (!(st > T(0))) {
        const T rV = T(kRV) * nu * (pl * b * f0 * ct);
        c[0] = c[1] = c[2] = c[3] = c[4] = c[5] = c[6] = T(0); c[7] = rV;
        return rV != T(0);
    }
    const T x = Te * hsqrt(T(1414.2135623730951) * st * b);
    const bool lo = x < T(120);
    const T q = lo ? x * T(1.0 / 120) : T(120) * hrcp(x);
    const T q2 = q * q, q4 = q2 * q2, q5 = q4 * q, q10 = q5 * q5, q20 = q10 * q10;
    const T s20 = hrcp(T(1) + q20), sw = lo ? q20 * s20 : s20;   // 0.5 + 0.5 tanh((ln x - ln 120) / 0.1)
    const T lx = hlog2(x + T(1e-16));
    const T ex = hexp(x * T(-1.0 / 47.2));
    const T extra = (T(0.011) * ex - T(7.9370052598409974e-01 / 67.44733739010397 * 3.141592653589793 * 1e4) * hexp2(fmin(T(-8.0 / 3) * lx, T(100)))) * sw;   // the bound: sw is zero long before
    const T jf = T(2.011) * hexp(hexp2(T(1.035) * lx) * T(-1.0 / 4.7)) - fcos(x * T(0.5)) * hexp(hexp2(T(1.2) * lx) * T(-1.0 / 2.73)) - T(0.011) * ex + extra;
    const T plb = pl * b;
    c[6] = T(0.5 * kRV) * nu * (jf * plb * b * (r[RW_KR] + T(6) * Te) * st * st);
    c[7] = T(kRV) * nu * (plb * (f0 * (T(1) - T(0.11) * hln(T(1) + T(0.035) * x))) * ct);
    const T nus = T(1.5) * nc * st * Te * Te + T(1);
    const T ls = hlog2(nu * hrcp(nus)) * T(1.0 / 3);             // of the cube root of nu / nu_s
    const T c13 = hexp2(-ls), c23 = c13 * c13;
    const T e13 = hexp(T(-1.8899) * hexp2(ls));
    constexpr double kJ = kEE * kEE / (2.0 * 1.7320508075688772 * kCL);   // times nu first: 2e-30 n_e underflows in FP32
    const T iT = hrcp(Te), pj = T(kJ) * nu * ne * iT * iT * e13;
    // j = pj f: the cap's ratios are the fits' own, whatever range pj is in
    const T fI = T(2.5651) * (T(1) + T(1.92) * c13 + T(0.9977) * c23);
    const T fQ = T(2.5651) * (T(1) + T(0.93193) * c13 + T(0.499873) * c23);
    const T fV = T(4.0 / 3) * iT * ct * hrcp(st) * (T(1.81384) * nus * inu + T(3.42319) * c23 + T(0.0292545) * hexp2(T(-1.5) * ls) + T(2.03773) * c13);
    const T jI = pj * fI, jQ = pj * fQ, jV = pj * fV, iI = hrcp(fI);
    // 1 / B_nu (planck): the series of exp(y) - 1 below 2e-3
    constexpr double kY = kHPL / (kME * kCL * kCL), kB = 2.0 * kHPL / (kCL * kCL);
    const T y = T(kY) * nu * iT;
    T em1;
    if (y < T(2e-3)) em1 = y * (T(1) + y * (T(0.5) + y * (T(1.0 / 6) + y * T(1.0 / 24))));
    else if constexpr (sizeof(T) == 4) em1 = expm1f(y);
    else em1 = expm1(y);
    const T iB = planck_inverse(T(kB * 1e33), nu, em1);
    const T cap = ratio_cap(fQ * iI, fV * iI);
    c[0] = jI; c[1] = jQ * cap; c[2] = jV * cap;
    c[3] = jI * iB; c[4] = c[1] * iB; c[5] = c[2] * iB;
    return jI > T(0) || c[6] != T(0) || c[7] != T(0);
}

// The power-law and kappa fits (powerlaw_cs, kappa_cs) from the row's constants, out of line: scenes that mix
// populations run them a population at a time. As there, a field along the ray is evaluated 1e-6 from the axis.
// lo: the low limit times its scale (n_e and nu_c first: the limit alone times the power underflows in FP32 at large kappa)
template <class T>
__device__ __forceinline__ T kappa_bridge(T lo, T arg, T ix) { return lo * hexp2(-ix * hlog2(T(1) + hexp2(arg))); }

template <class T>
__device__ __noinline__ bool other_row(const T* r, int kind, T ne, T nu, T st, T ct, T* c) {
    st = fmax(st, T(1e-6));
    const T* e = r + RW_E;
    const T nc = r[RW_NUC], nb = nc * st, inu = hrcp(nu), ist = hrcp(st), ls = hlog2(st);
    const T sg = ct > T(0) ? T(1) : (ct < T(0) ? T(-1) : T(0));
    T jI, jQ, jV, aI, aQ, aV, rQ, rV;
    if (kind == KS_POWERLAW22) {
        const T xx = nu * hrcp(nb), lx = hlog2(xx), ix = hrsqrt(xx);
        const T pw = hexp2(-e[EP_P1] * lx);                      // xx^(-(p - 1) / 2)
        jI = ne * nb * e[EP_J] * pw;
        jQ = e[EP_JQ] * jI;
        jV = e[EP_JV] * ct * ist * ix * jI;
        aI = ne * inu * e[EP_A] * pw * ix * ix * ix;             // xx^(-(p + 2) / 2)
        aQ = e[EP_AQ] * aI;
        const T t6 = T(31.0 / 10) * hexp2(T(-48.0 / 25) * ls) - T(31.0 / 10);
        aV = t6 > T(0) ? e[EP_AV] * hexp2(T(64.0 / 125) * hlog2(t6)) * ix * sg * aI : T(0);
        rQ = ne * e[EP_RQ] * (nb * inu) * (nb * inu) * inu * (T(1) - hexp2(e[EP_PG] - e[EP_PH] * lx));
        rV = ne * e[EP_RV] * nb * inu * inu * ct * ist;
    } else {
        const T X = nu * hrcp(nb) * e[EK_X], lx = hlog2(X);
        const T pj = ne * nb * hexp2(T(1.0 / 3) * lx), pa = ne * hrcp(nb) * hexp2(T(-5.0 / 3) * lx);
        jI = kappa_bridge(pj * e[EK_I], e[EK_I + 1] * lx + e[EK_I + 2], e[EK_I + 3]);
        jQ = kappa_bridge(pj * e[EK_Q], e[EK_Q + 1] * lx + e[EK_Q + 2], e[EK_Q + 3]);
        aI = kappa_bridge(pa * e[EK_AI], e[EK_AI + 1] * lx + e[EK_AI + 2], e[EK_AI + 3]);
        aQ = kappa_bridge(pa * e[EK_AQ], e[EK_AQ + 1] * lx + e[EK_AQ + 2], e[EK_AQ + 3]);
        // circular: the limits carry (sin^-u - 1)^v and X^-0.35 against X^-0.5
        const T u1 = hexp2(T(-12.0 / 5) * ls) - T(1), u2 = hexp2(T(-2.5) * ls) - T(1);
        const T u3 = hexp2(T(-114.0 / 50) * ls) - T(1), u4 = hexp2(T(-41.0 / 20) * ls) - T(1);
        const T x35 = hexp2(T(-7.0 / 20) * lx);
        jV = aV = T(0);
        if (u1 > T(0) && u2 > T(0)) {
            const T l1 = T(12.0 / 25) * hlog2(u1), l2 = T(11.0 / 25) * hlog2(u2);
            jV = sg * kappa_bridge(pj * x35 * e[EK_V] * hexp2(l1), e[EK_V + 3] * (e[EK_V + 1] * lx + e[EK_V + 2] + l1 - l2 + T(3.0 / 20) * lx), e[EK_V + 4]);
        }
        if (u3 > T(0) && u4 > T(0)) {
            const T l3 = T(223.0 / 500) * hlog2(u3), l4 = T(0.5) * hlog2(u4);
            aV = sg * kappa_bridge(pa * x35 * e[EK_AV] * hexp2(l3), e[EK_AV + 3] * (e[EK_AV + 1] * lx + e[EK_AV + 2] + l3 - l4 + T(3.0 / 20) * lx), e[EK_AV + 4]);
        }
        const int i = int(e[EK_FIT]);
        auto fit_q = [&](int n) {
            const T k84 = n == 0 ? T(1.0 / 30) : n == 1 ? T(1.0 / 18) : n == 2 ? T(1.0 / 12) : T(1.0 / 8);
            const T ks_ = n == 0 ? T(1.0 / 10) : n == 1 ? T(1.0 / 6) : n == 2 ? T(1.0 / 4) : T(3.0 / 8);
            const T kx = n == 0 ? T(1.5) : n == 1 ? T(1.75) : n == 2 ? T(2) : T(2.25);
            const T kp = n == 0 ? T(0.471) : n == 1 ? T(0.5) : n == 2 ? T(0.525) : T(0.541);
            T s, cs;
            sincos_product(fmin(X, T(1e6)), ks_, s, cs);   // beyond, its factor has vanished
            return T(1) - hexp(-k84 * hexp2(T(0.84) * lx)) - s * hexp(-kx * hexp2(kp * lx));
        };
        auto fit_v = [&](int n) {
            const T k = n == 0 ? T(0.447) : n == 1 ? T(0.391) : n == 2 ? T(0.348) : T(0.313);
            return T(1) - T(0.17) * hln(T(1) + k * hexp2(T(-0.5) * lx));
        };
        rQ = ne * (nb * inu) * (nb * inu) * inu * (e[EK_FQ0] * fit_q(i) + e[EK_FQ1] * fit_q(i + 1));
        rV = ne * nc * ct * inu * inu * (e[EK_FV0] * fit_v(i) + e[EK_FV1] * fit_v(i + 1));
    }
    const T fe = row_cap(jI, jQ, jV), fa = row_cap(aI, aQ, aV);
    c[0] = jI; c[1] = jQ * fe; c[2] = jV * fe; c[3] = aI; c[4] = aQ * fa; c[5] = aV * fa; c[6] = rQ; c[7] = rV;
    return jI > T(0) || aI > T(0) || rQ != T(0) || rV != T(0);
}

// 2^floor(log2 v) of a normal positive v (the exponent alone), 1 otherwise
__device__ __forceinline__ float pow2_of(float v) {
    const int e = __float_as_int(v) & 0x7f800000;
    return (v > 0.f && e != 0 && e != 0x7f800000) ? __int_as_float(e) : 1.f;
}
__device__ __forceinline__ double pow2_of(double v) {
    const long long e = __double_as_longlong(v) & 0x7ff0000000000000ll;
    return (v > 0.0 && e != 0 && e != 0x7ff0000000000000ll) ? __longlong_as_double(e) : 1.0;
}

// K v with K = [0 aQ aU aV; aQ 0 rV -rU; aU -rV 0 rQ; aV rU -rQ 0], k = (aQ, aU, aV, rQ, rU, rV)
template <class T>
__device__ __forceinline__ void kvec(const T k[6], const T v[4], T o[4]) {
    o[0] = k[0] * v[1] + k[1] * v[2] + k[2] * v[3];
    o[1] = k[0] * v[0] + k[5] * v[2] - k[4] * v[3];
    o[2] = k[1] * v[0] - k[5] * v[1] + k[3] * v[3];
    o[3] = k[2] * v[0] + k[4] * v[1] - k[3] * v[2];
}
// v K (a row vector)
template <class T>
__device__ __forceinline__ void kvec_t(const T k[6], const T v[4], T o[4]) {
    o[0] = k[0] * v[1] + k[1] * v[2] + k[2] * v[3];
    o[1] = k[0] * v[0] - k[5] * v[2] + k[4] * v[3];
    o[2] = k[1] * v[0] + k[5] * v[1] - k[3] * v[3];
    o[3] = k[2] * v[0] - k[4] * v[1] + k[3] * v[2];
}

// M_n(a) = int_0^1 t^n e^{-at} dt, n = 0..9 (step.jl:239-268). |a| < 1: the series of M_9 (twelve terms reach
// FP32's rounding, 24 FP64's) and the downward recurrence M_{n-1} = (a M_n + e^{-a}) / n, which scales an error by
// |a| / n; past it the upward one.
template <class T>
__device__ __forceinline__ void step_moments(const MomentCoeffs& MC, T a, T ex, T M[10]) {
    if (fabs(a) < T(1)) {
        constexpr int K = sizeof(T) == 4 ? 11 : 23;
        T s = mcoef<T>(MC, 9, K);
#pragma unroll
        for (int m = K - 1; m >= 0; --m) s = fma(a, s, mcoef<T>(MC, 9, m));
        M[9] = s;
#pragma unroll
        for (int n = 9; n >= 1; --n) M[n - 1] = fma(a, M[n], ex) * T(1.0 / n);
    } else {
        const T ia = hrcp(a);
        M[0] = (T(1) - ex) * ia;
#pragma unroll
        for (int n = 1; n < 10; ++n) M[n] = (T(n) * M[n - 1] - ex) * ia;
    }
}
// (1 - e^{-x}) / x
template <class T>
__device__ __forceinline__ T step_phi(T x) {
    if (fabs(x) < (sizeof(T) == 4 ? T(1) : T(0.1)))   // FP32: no cancellation; FP64 has expm1
        return T(1) - x * T(0.5) * (T(1) - x * T(1.0 / 3) * (T(1) - x * T(0.25) * (T(1) - x * T(0.2) * (T(1) - x * T(1.0 / 6) * (T(1) - x * T(1.0 / 7) *
               (T(1) - x * T(0.125) * (T(1) - x * T(1.0 / 9) * (T(1) - x * T(0.1) * (T(1) - x * T(1.0 / 11))))))))));
    if constexpr (sizeof(T) == 4) return (T(1) - hexp(-x)) * hrcp(x);
    else return -expm1(-x) / x;
}

// step_coefficients of a value (no duals): the coefficients (o_n, e_n) at the scaled invariants, the same branches
// and thresholds, sinh and cosh below b_1 = 1 from their series.
template <class T>
__device__ __forceinline__ void step_scalars(const MomentCoeffs& MC, T a, T a2, T r2, T ar, T D, T o[4], T e[4]) {
    const T ex = hexp(-a);
    T M[10];
    step_moments(MC, a, ex, M);
    const T h = (a2 - r2) * T(0.5), rt2 = h * h + ar * ar;
    const T root = rt2 > T(0) ? hsqrt(rt2) : T(0);
    const T big = fabs(h) + root, small = big > T(0) ? ar * ar * hrcp(big) : T(0);
    const T L1sq = h >= T(0) ? big : small, L2sq = h >= T(0) ? small : big, Th = L1sq + L2sq, D2 = D * D;
    if ((a2 + r2) * D2 < lin_thr<T>()) {
        o[0] = ex; o[1] = -D * ex; o[2] = T(0); o[3] = T(0);
        e[0] = D * M[0]; e[1] = -D2 * M[1]; e[2] = T(0); e[3] = T(0);
        return;
    }
    if (Th * D2 * ((a2 + r2) * D2 + T(1)) < cub_thr<T>()) {
        o[0] = ex; o[1] = -D * ex; o[2] = (D2 * T(0.5)) * ex; o[3] = -(D2 * D * T(1.0 / 6)) * ex;
        e[0] = D * M[0]; e[1] = -D2 * M[1]; e[2] = (D2 * D * T(0.5)) * M[2]; e[3] = -(D2 * D2 * T(1.0 / 6)) * M[3];
        return;
    }
    const T b1 = L1sq > T(0) ? hsqrt(L1sq) * D : T(0), b2 = L2sq > T(0) ? hsqrt(L2sq) * D : T(0);
    const T b1s = b1 * b1, b2s = b2 * b2;
    T chm1, shc;   // e^{-a} (cosh b1 - 1), e^{-a} sinh(b1) / b1
    T icoshm1, ishx;   // the integrals of cosh(b1 t) - 1 and of sinh(b1 t) / b1 - t under e^{-at}
    if (b1 < T(1)) {
        chm1 = ex * (b1s * T(0.5) * (T(1) + b1s * T(1.0 / 12) * (T(1) + b1s * T(1.0 / 30) * (T(1) + b1s * T(1.0 / 56) * (T(1) + b1s * T(1.0 / 90) *
               (T(1) + b1s * T(1.0 / 132) * (T(1) + b1s * T(1.0 / 182))))))));
        shc = ex * (T(1) + b1s * T(1.0 / 6) * (T(1) + b1s * T(1.0 / 20) * (T(1) + b1s * T(1.0 / 42) * (T(1) + b1s * T(1.0 / 72) *
              (T(1) + b1s * T(1.0 / 110) * (T(1) + b1s * T(1.0 / 156) * (T(1) + b1s * T(1.0 / 210))))))));
    } else {
        const T em = hexp(b1 - a), ep = hexp(-(a + b1));
        chm1 = (em + ep) * T(0.5) - ex;
        shc = (em - ep) * T(0.5) * hrcp(b1);
    }
    const T ph_a = M[0];
    if (b1 < T(0.1)) {
        icoshm1 = b1s * (M[2] * T(0.5) + b1s * (M[4] * T(1.0 / 24) + b1s * (M[6] * T(1.0 / 720) + b1s * M[8] * T(1.0 / 40320))));
        ishx = b1s * (M[3] * T(1.0 / 6) + b1s * (M[5] * T(1.0 / 120) + b1s * (M[7] * T(1.0 / 5040) + b1s * M[9] * T(1.0 / 362880))));
    } else {
        const T pm = step_phi(a - b1), pp = step_phi(a + b1);
        icoshm1 = (pm + pp) * T(0.5) - ph_a;
        ishx = (pm - pp) * T(0.5) * hrcp(b1) - M[1];
    }
    // one sine and cosine of the half angle: sin b2 = 2 s c, 1 - cos b2 = 2 s^2
    T sh2, ch2;
    fsincos(b2 * T(0.5), sh2, ch2);
    const T sb2 = T(2) * sh2 * ch2, vers = T(2) * sh2 * sh2, cb2 = T(1) - vers;
    T sincb2, iversin, icos, isinc;
    if (b2 < T(0.1)) {
        sincb2 = T(1) - b2s * T(1.0 / 6) * (T(1) - b2s * T(1.0 / 20) * (T(1) - b2s * T(1.0 / 42) * (T(1) - b2s * T(1.0 / 72) * (T(1) - b2s * T(1.0 / 110)))));
        iversin = b2s * (M[2] * T(0.5) - b2s * (M[4] * T(1.0 / 24) - b2s * (M[6] * T(1.0 / 720) - b2s * M[8] * T(1.0 / 40320))));
        icos = ph_a - iversin;
        isinc = M[1] - b2s * (M[3] * T(1.0 / 6) - b2s * (M[5] * T(1.0 / 120) - b2s * (M[7] * T(1.0 / 5040) - b2s * M[9] * T(1.0 / 362880))));
    } else {
        const T ib2 = hrcp(b2), id = hrcp(a * a + b2s);
        sincb2 = sb2 * ib2;
        icos = (a - ex * (a * cb2 - b2 * sb2)) * id;
        iversin = ph_a - icos;
        isinc = (T(1) - ex * (a * sincb2 + cb2)) * id;
    }
    const T iTh = hrcp(Th);
    const T so = D * shc, sn = D * ex * sincb2, Is = D2 * isinc, Ish = D2 * (M[1] + ishx);
    o[0] = (L2sq * (chm1 + ex) + L1sq * ex * cb2) * iTh;
    o[1] = -(so * L2sq + sn * L1sq) * iTh;
    o[2] = (chm1 + ex * vers) * iTh;
    o[3] = (sn - so) * iTh;
    e[0] = D * (L2sq * (ph_a + icoshm1) + L1sq * icos) * iTh;
    e[1] = -(Ish * L2sq + Is * L1sq) * iTh;
    e[2] = D * (icoshm1 + iversin) * iTh;
    e[3] = (Is - Ish) * iTh;
}

// A step record: o_0..3, E, the six entries of the rescaled K, the active flag (transfer_step
// without its matrices).
constexpr int kRec = 16;
template <class T>
__device__ __forceinline__ void step_record(const MomentCoeffs& MC, const T v[11], T Dl, T rec[kRec]) {
    const T s = pow2_of(Dl), D = Dl / s;
    T k[6], o[4], e[4];
#pragma unroll
    for (int q = 0; q < 6; ++q) k[q] = v[5 + q] * s;
    step_scalars(MC, v[4] * s * D, k[0] * k[0] + k[1] * k[1] + k[2] * k[2], k[3] * k[3] + k[4] * k[4] + k[5] * k[5],
                 k[0] * k[3] + k[1] * k[4] + k[2] * k[5], D, o, e);
    T j1[4], j2[4], j3[4];
    kvec(k, v, j1); kvec(k, j1, j2); kvec(k, j2, j3);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        rec[q] = o[q];
        rec[4 + q] = s * (e[0] * v[q] + e[1] * j1[q] + e[2] * j2[q] + e[3] * j3[q]);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) rec[8 + q] = k[q];
    rec[14] = T(1);
    rec[15] = T(0);
}

// 16-byte moves of n values between registers and shared or global memory
template <int N>
__device__ __forceinline__ void put16(float* p, const float* v) {
#pragma unroll
    for (int q = 0; q < N; q += 4) *reinterpret_cast<float4*>(p + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
}
template <int N>
__device__ __forceinline__ void put16(double* p, const double* v) {
#pragma unroll
    for (int q = 0; q < N; q += 2) *reinterpret_cast<double2*>(p + q) = make_double2(v[q], v[q + 1]);
}
template <int N>
__device__ __forceinline__ void get16(const float* p, float* v) {
#pragma unroll
    for (int q = 0; q < N; q += 4) {
        const float4 f = *reinterpret_cast<const float4*>(p + q);
        v[q] = f.x; v[q + 1] = f.y; v[q + 2] = f.z; v[q + 3] = f.w;
    }
}
template <int N>
__device__ __forceinline__ void get16(const double* p, double* v) {
#pragma unroll
    for (int q = 0; q < N; q += 2) {
        const double2 f = *reinterpret_cast<const double2*>(p + q);
        v[q] = f.x; v[q + 1] = f.y;
    }
}

// ---- candidates ------------------------------------------------------------------------------------------

// Whether row r's support can reach the box at the observation time: the circle, then the arc, that the centre runs
// on, or a knot splat's bounding sphere. The box and this test are FP32 in either precision. The box holds lookback
// times and the phase is formed from t_obs - t0, taken in T, so that what is rounded are differences of times: in FP32
// a time of 1e7 is off by 0.5. Positions are padded by a few of their roundings.
template <class T>
__device__ __forceinline__ bool row_reaches(const T* r, const UnitBox& b, T t_obs) {
    const float cz = float(r[RW_CZ]), rho = float(r[RW_RHO]);
    if (int(r[RW_KIND]) == KS_KNOT21) {
        const float cx = float(r[RW_CX]), cy = float(r[RW_CY]), e = 1e-6f * (fabsf(cx) + fabsf(cy) + fabsf(cz));
        const float dx = fmaxf(fmaxf(b.xlo - cx, cx - b.xhi) - e, 0.f);
        const float dy = fmaxf(fmaxf(b.ylo - cy, cy - b.yhi) - e, 0.f);
        const float dz = fmaxf(fmaxf(b.zlo - cz, cz - b.zhi) - e, 0.f);
        return dx * dx + dy * dy + dz * dz <= rho * 1.0001f;
    }
    const float supp = float(r[RW_SUPP]) * 1.0001f, e = 1e-6f * (rho + fabsf(cz));
    const float dr = fmaxf(fmaxf(b.rlo - rho, rho - b.rhi) - e, 0.f);
    const float dz = fmaxf(fmaxf(b.zlo - cz, cz - b.zhi) - e, 0.f);
    if (!(dr * dr + dz * dz <= supp)) return false;
    const float om = float(r[RW_OMEGA]), off = float(t_obs - r[RW_T0]);
    const float pa = om * (off - b.shi), pb = om * (off - b.slo);
    // the pad covers the FP32 rounding of the angles (phases up to ~1e3 rad) and positions, and in FP32 that of the
    // times a sample is tested at
    float pad = 1e-3f * rho + 1e-4f * (fabsf(pa) + fabsf(pb)) * rho + 1e-3f;
    if (sizeof(T) == 4) pad += 2.4e-7f * fabsf(om) * rho * (fabsf(float(t_obs)) + fabsf(float(r[RW_T0])));
    const float lo = fminf(pa, pb), hi = fmaxf(pa, pb);
    if (!(b.slo <= b.shi) || !(hi - lo < 6.0f)) return true;
    const float A = float(r[RW_ANG]) + lo, B = float(r[RW_ANG]) + hi;
    float sa, ca, sb, cb;
    sincosf(A, &sa, &ca);
    sincosf(B, &sb, &cb);
    float xlo = rho * fminf(ca, cb), xhi = rho * fmaxf(ca, cb), ylo = rho * fminf(sa, sb), yhi = rho * fmaxf(sa, sb);
    // the axis directions 0, pi/2, pi, 3 pi/2 (+ 2 pi k) inside [A, B] (with a margin: conservative)
    const float i2pi = 0.15915494309189535f, m = 1e-3f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float d = q * 1.5707963267948966f;
        const float k = ceilf((A - m - d) * i2pi - 1e-6f);
        if (d + 6.283185307179586f * k <= B + m) {
            if (q == 0) xhi = rho;
            else if (q == 1) yhi = rho;
            else if (q == 2) xlo = -rho;
            else ylo = -rho;
        }
    }
    const float dx = fmaxf(fmaxf(b.xlo - (xhi + pad), (xlo - pad) - b.xhi), 0.f);
    const float dy = fmaxf(fmaxf(b.ylo - (yhi + pad), (ylo - pad) - b.yhi), 0.f);
    return dx * dx + dy * dy + dz * dz <= supp;
}

// ---- the kernel ------------------------------------------------------------------------------------------

template <class T, int CH, int KM, int NT>
struct TransportSmem {
    static constexpr int W = NT / 32, ST = row_stride<T, KM>();
    static constexpr int REC = CH * kRec + 16 / int(sizeof(T));   // an odd number of 16-byte words per sample
    __host__ __device__ static size_t rows_bytes(int ntot, int nkv) { return ((size_t(ntot) * ST + nkv) * sizeof(T) + 15) / 16 * 16; }
    __host__ __device__ static size_t bytes(int ntot, int nkv, int run, int cap, bool rows_shared) {
        const int nw = (ntot + 31) / 32;
        return (rows_shared ? rows_bytes(ntot, nkv) : 0) + size_t(cap) * REC * sizeof(T) + 5 * 32 * sizeof(T)   // rows, records, ray constants
               + size_t(run) * 32 * nw * 4 + size_t(nw) * (W + 3) * 4                                            // masks, candidates, populations
               + W * 10 * 4 + run * 8 + 64 * 4 + size_t(cap) * 4 + 64;                                           // boxes, lane masks, bins, orders
    }
};

template <class T, int CH, int KM, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
k_transport(PlanView P, Spacetime st, TransportJob job, const T* __restrict__ rows_g, const double* __restrict__ ct,
            const double* __restrict__ cnu, const T* __restrict__ stream, unsigned long long* __restrict__ work, T* __restrict__ seg_out,
            unsigned long long* __restrict__ counters, unsigned* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem[];
    using SM = TransportSmem<T, CH, KM, NT>;
    constexpr int W = NT / 32, ST = SM::ST, REC = SM::REC;
    constexpr int NTASK = (4 * CH + W - 1) / W;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntot = job.ntot, nw = (ntot + 31) >> 5, R = job.run, RS = R / W, cap = job.cap;
    // the splat rows and knots into shared memory by one bulk copy (FP64 tables past its size stay in global memory)
    unsigned char* at = smem;
    const T* rows = rows_g;
    if (job.rows_shared) {
        __shared__ __align__(8) unsigned long long bar;
        const unsigned bytes = unsigned(SM::rows_bytes(ntot, job.nkv));
        if (bytes > 0 && !stage_bulk(smem, rows_g, bytes, &bar, job.stage_test == 0, job.stage_test ? 4096 : kStageWaitLimit)) {
            if (tid == 0) atomicOr(err, 1u);
            return;
        }
        rows = reinterpret_cast<const T*>(smem);
        at += bytes;
    }
    const T* knots = rows + (long long)ntot * ST;
    T* rec = reinterpret_cast<T*>(at);                                   // [cap][REC]
    T* rayc = rec + (long long)cap * REC;                                // [5][32]: alpha, beta, eta, lambda, dtau
    unsigned* masks = reinterpret_cast<unsigned*>(rayc + 5 * 32);        // [run][nw][32]
    unsigned* cand = masks + R * nw * 32;                                // [W][nw]
    unsigned* kinds = cand + W * nw;                                     // [3][nw]: the splats of each population
    float* boxes = reinterpret_cast<float*>(kinds + 3 * nw);             // [W][10]
    unsigned* ball = reinterpret_cast<unsigned*>(boxes + W * 10);        // [run]: the rays with a passing splat
    int* base = reinterpret_cast<int*>(ball + R);                        // [run]: records before the sample
    int* bins = base + R;                                                // [64]
    unsigned short* order = reinterpret_cast<unsigned short*>(bins + 64);   // [cap]: sample << 5 | lane, by number of splats
    unsigned short* order2 = order + cap;                                   // ... and by record
    __shared__ unsigned long long s_unit;
    __shared__ float s_reach;
    // the table's reach (table_reach2) and its populations
    if (tid == 0) s_reach = 0.f;
    for (int q = tid; q < 3 * nw; q += NT) kinds[q] = 0u;
    __syncthreads();
    {
        float m = 0.f;
        for (int i = tid; i < ntot; i += NT) {
            const T* r = rows + (long long)i * ST;
            const int kind = int(r[RW_KIND]);
            const float cx = float(r[RW_CX]), cy = float(r[RW_CY]), cz = float(r[RW_CZ]);
            m = fmaxf(m, sqrtf(cx * cx + cy * cy + cz * cz) + sqrtf(float(kind == KS_KNOT21 ? r[RW_RHO] : r[RW_SUPP])));
            if (KM != 1) atomicOr(&kinds[(kind == KS_POWERLAW22 ? 1 : kind == KS_KAPPA22 ? 2 : 0) * nw + (i >> 5)], 1u << (i & 31));
        }
        atomicMax(reinterpret_cast<int*>(&s_reach), __float_as_int(m));
    }
    __syncthreads();
    const float reach = s_reach * 1.001f + 1e-3f;
    const T reach2 = T(reach) * T(reach);
    const T a = T(st.a), a_sin_tho = T(st.a * sin(st.thetao));
    T* gstate = static_cast<T*>(job.gstate);
    const int N = st.N;
    const long long npad = job.npad, fs = npad;   // a field's stride in the stream
    unsigned ev[7] = {0, 0, 0, 0, 0, 0, 0};
    const int per_chunk = job.nseg * job.nframes * job.nvc;
    const long long total = job.nchunks * per_chunk;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_unit = atomicAdd(work, 1ull);
        __syncthreads();
        if (s_unit >= (unsigned long long)total) break;
        const long long u = total - 1 - (long long)s_unit;   // the last rays first: they carry most of the work
        const long long jb = u / per_chunk * 32;
        const int rem = int(u % per_chunk), seg = rem / (job.nframes * job.nvc), y = rem % (job.nframes * job.nvc);
        const int f = y / job.nvc, v0 = (y % job.nvc) * CH, nc = min(CH, job.nfreq - v0);
        const bool live = jb + lane < job.npix;
        const long long jl = live ? jb + lane : job.npix - 1, jp = job.j0 + jl;   // in the stream, in the plan
        const int k0 = 1 + seg * job.seg_len, nsamp = live ? int(P.get(PF_NSAMP, jp)) : 0;
        int klim = nsamp;
        if (job.kstop && live) klim = min(klim, job.kstop[jp] - 1);
        const int k1 = min(k0 + job.seg_len, __reduce_max_sync(0xffffffffu, klim) + 1);
        if (warp == 0) {
            rayc[lane] = T(P.get(PF_ALPHA, jp)); rayc[32 + lane] = T(P.get(PF_BETA, jp)); rayc[64 + lane] = T(P.get(PF_ETA, jp));
            rayc[96 + lane] = T(P.get(PF_LAM, jp)); rayc[128 + lane] = T(P.get(PF_DTAU, jp));
            ev[0] += unsigned(max(0, min(nsamp + 1, k0 + job.seg_len) - k0)) * nc;
        }
        const T t_obs = T(ct[f]);
        T nu[CH], Lnu[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const double v = cnu[min(v0 + c, job.nfreq - 1)];
            nu[c] = T(v);
            Lnu[c] = T(job.L / (v / kNU0));
        }
        // this thread's rows of P and entries of S: task = (frequency, row)
        T pr[NTASK][4], ps[NTASK];
#pragma unroll
        for (int q = 0; q < NTASK; ++q) {
            const int row = (q * W + warp) & 3;
#pragma unroll
            for (int s = 0; s < 4; ++s) pr[q][s] = s == row ? T(1) : T(0);
            ps[q] = T(0);
        }
        for (int kr = k0; kr < k1; kr += R) {
            const T* sp = stream + (long long)(kr - 1) * SM_COUNT * npad + jl;
            // 1. the candidates of the run's sixteen-sample groups (a group's warps share the words), then the tests
            {
                UnitBox b = unit_box_empty();
                for (int s = 0; s < RS; ++s) {
                    const int kl = warp * RS + s;
                    if (kr + kl > klim || kr + kl >= k1) break;
                    const T* p = sp + (long long)kl * SM_COUNT * fs;
                    if (!(stream_flags(p[SM_FLAGS * fs]) & 8u)) continue;
                    const T x = p[SM_X * fs], yy = p[SM_Y * fs], z = p[SM_Z * fs];
                    if (x * x + yy * yy + z * z > reach2) continue;   // beyond every splat: no candidate needed
                    unit_box_add(b, float(x), float(yy), float(z), float(p[SM_T * fs]));
                }
                unit_box_reduce(b);
                const float* bf = reinterpret_cast<const float*>(&b);
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 10; ++q) boxes[warp * 10 + q] = bf[q];
            }
            __syncthreads();
            {
                const int G = max(1, min(W, 16 / RS)), g0 = warp / G * G;
                UnitBox b = unit_box_empty();
                for (int q = g0; q < g0 + G; ++q) {
                    const float* o = boxes + q * 10;
                    b.xlo = fminf(b.xlo, o[0]); b.xhi = fmaxf(b.xhi, o[1]); b.ylo = fminf(b.ylo, o[2]); b.yhi = fmaxf(b.yhi, o[3]);
                    b.zlo = fminf(b.zlo, o[4]); b.zhi = fmaxf(b.zhi, o[5]); b.rlo = fminf(b.rlo, o[6]); b.rhi = fmaxf(b.rhi, o[7]);
                    b.slo = fminf(b.slo, o[8]); b.shi = fmaxf(b.shi, o[9]);
                }
                for (int wd = warp - g0; wd < nw; wd += G) {
                    const int i = wd * 32 + lane;
                    const bool keep = i < ntot && b.xlo <= b.xhi && row_reaches(rows + (long long)i * ST, b, t_obs);
                    const unsigned m = __ballot_sync(0xffffffffu, keep);
                    if (lane == 0) cand[g0 / G * nw + wd] = m;
                }
            }
            __syncthreads();
            {
                const int G = max(1, min(W, 16 / RS));
                const unsigned* cw = cand + warp / G * nw;
                for (int s = 0; s < RS; ++s) {
                    const int kl = warp * RS + s;
                    const T* p = sp + (long long)kl * SM_COUNT * fs;
                    bool test = kr + kl <= klim && kr + kl < k1;
                    T x = T(0), yy = T(0), z = T(0), t = T(0), rho = T(0);
                    if (test) test = (stream_flags(p[SM_FLAGS * fs]) & 8u) != 0u;
                    if (test) {
                        ev[1]++;
                        x = p[SM_X * fs]; yy = p[SM_Y * fs]; z = p[SM_Z * fs];
                        test = x * x + yy * yy + z * z <= reach2;
                        t = t_obs - p[SM_T * fs];
                        rho = sqrt(x * x + yy * yy);
                    }
                    unsigned any = 0u;
                    for (int wd = 0; wd < nw; ++wd) {
                        unsigned m = 0u, c = cw[wd];
                        while (c) {   // the same splats for the whole warp
                            const int b = __ffs(c) - 1;
                            c &= c - 1;
                            const T* r = rows + (long long)(wd * 32 + b) * ST;
                            if (!test) continue;
                            ev[2]++;
                            T q;
                            if (KM == 1 || int(r[RW_KIND]) != KS_KNOT21) {
                                // farther from the circle the centre runs on than the support: outside at every time
                                const T dr = rho - r[RW_RHO], dz = z - r[RW_CZ];
                                if (dr * dr + dz * dz > r[RW_SUPP]) continue;
                                if (!row_exponent<true>(r, t, x, yy, z, q)) continue;
                            } else {
                                const T dx = x - r[RW_CX], dy = yy - r[RW_CY], dz = z - r[RW_CZ];
                                if (dx * dx + dy * dy + dz * dz > r[RW_RHO]) continue;   // outside the knots' bounding sphere
                                row_knot_exponent(r, knots, t, x, yy, z, q);
                            }
                            ev[3]++;
                            if (q < T(kQCUT)) m |= 1u << b;
                        }
                        masks[(kl * nw + wd) * 32 + lane] = m;
                        any |= m;
                    }
                    const unsigned bl = __ballot_sync(0xffffffffu, any != 0u);
                    if (lane == 0) ball[kl] = bl;
                }
            }
            __syncthreads();
            // 2. and 3. in windows of whole samples (all rays) whose records fit
            for (int w0 = 0; w0 < R;) {
                int w1 = w0, n = 0;
                for (; w1 < R; ++w1) {
                    const int c = __popc(ball[w1]);
                    if (n + c > cap) break;
                    if (tid == 0) base[w1] = n;
                    n += c;
                }
                if (n == 0) { w0 = w1; continue; }   // every thread sees the same counts
                if (tid < 33) bins[tid] = 0;
                __syncthreads();
                // the samples in descending order of their number of splats (a counting sort; equal counts in any order)
                for (int kl = w0 + warp; kl < w1; kl += W) {
                    if (!((ball[kl] >> lane) & 1u)) continue;
                    int m = 0;
                    for (int wd = 0; wd < nw; ++wd) m += __popc(masks[(kl * nw + wd) * 32 + lane]);
                    atomicAdd(&bins[32 - min(m, 32)], 1);
                }
                __syncthreads();
                if (warp == 0) {
                    const int v = bins[lane];
                    int incl = v;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int o = __shfl_up_sync(0xffffffffu, incl, d);
                        if (lane >= d) incl += o;
                    }
                    bins[lane] = incl - v;
                }
                __syncthreads();
                for (int kl = w0 + warp; kl < w1; kl += W) {
                    if (!((ball[kl] >> lane) & 1u)) continue;
                    int m = 0;
                    for (int wd = 0; wd < nw; ++wd) m += __popc(masks[(kl * nw + wd) * 32 + lane]);
                    order[atomicAdd(&bins[32 - min(m, 32)], 1)] = (unsigned short)(kl << 5 | lane);
                }
                __syncthreads();
                // 2. evaluation: chunks of 32 samples to the warps, back and forth (longest first)
                for (int rd = 0; rd * NT < n; ++rd) {
                    const int i = (rd * W + ((rd & 1) ? W - 1 - warp : warp)) * 32 + lane;
                    if (i >= n) continue;
                    const int kl = order[i] >> 5, o = order[i] & 31;
                    const long long jo = jb + o;
                    const T* p = stream + (long long)(kr + kl - 1) * SM_COUNT * npad + jo;
                    const T x = p[SM_X * fs], yy = p[SM_Y * fs], z = p[SM_Z * fs], t = t_obs - p[SM_T * fs];
                    const T r = p[SM_R * fs], sth = p[SM_STH * fs], cth = p[SM_CTH * fs];
                    const unsigned fl = stream_flags(p[SM_FLAGS * fs]);
                    const T alpha = rayc[o], beta = rayc[32 + o];
                    const SampleFrame<T> F = sample_frame(a, r, T(0), sth, cth, rayc[64 + o], rayc[96 + o], (fl & 2u) != 0u, (fl & 4u) != 0u);
                    T acc[CH][11];
                    unsigned act = 0u;
#pragma unroll
                    for (int c = 0; c < CH; ++c)
#pragma unroll
                        for (int q = 0; q < 11; ++q) acc[c][q] = T(0);
#pragma unroll 1
                    for (int pass = 0; pass < (KM == 1 ? 1 : 3); ++pass)
#pragma unroll 1
                        for (int wd = 0; wd < nw; ++wd) {
                            unsigned m = masks[(kl * nw + wd) * 32 + o];
                            if (KM != 1) m &= kinds[pass * nw + wd];
                            while (m) {
                                const int b = __ffs(m) - 1;
                                m &= m - 1;
                                const T* sr = rows + (long long)(wd * 32 + b) * ST;
                                T q;
                                if (KM == 1 || int(sr[RW_KIND]) != KS_KNOT21) row_exponent<false>(sr, t, x, yy, z, q);
                                else row_knot_exponent(sr, knots, t, x, yy, z, q);
                                const T ne = sr[RW_NE] * weight_of(q);
                                const LFrame<T> lf = row_frame(F, sr, alpha, beta, a_sin_tho);
                                T sb, cb;
                                pitch_sc(lf.cosB, sb, cb);
                                ev[5]++;
#pragma unroll
                                for (int c = 0; c < CH; ++c) {
                                    if (c >= nc) break;
                                    const T nuf = nu[c] * lf.g;
                                    T cf[8];
                                    const bool on = (KM == 1 || pass == 0) ? thermal_row(sr, ne, nuf, sb, cb, cf)
                                                                           : other_row(sr, pass == 1 ? KS_POWERLAW22 : KS_KAPPA22, ne, nuf, sb, cb, cf);
                                    if (!on) continue;
                                    act |= 1u << c;
                                    const T nh = nuf * T(1.0 / kNU0), i2 = T(1) / (nh * nh);
                                    const T jQ = cf[1] * i2, aQ = cf[4] * nh, rQ = cf[6] * nh;
                                    acc[c][0] += cf[0] * i2; acc[c][1] += jQ * lf.c2c; acc[c][2] += jQ * lf.s2c; acc[c][3] += cf[2] * i2;
                                    acc[c][4] += nh * cf[3]; acc[c][5] += aQ * lf.c2c; acc[c][6] += aQ * lf.s2c; acc[c][7] += cf[5] * nh;
                                    acc[c][8] += rQ * lf.c2c; acc[c][9] += rQ * lf.s2c; acc[c][10] += nh * cf[7];
                                }
                            }
                        }
                    const int id = base[kl] + __popc(ball[kl] & ((1u << o) - 1u));
                    const T sgd = (r * r + a * a * cth * cth) * rayc[128 + o];   // Sigma dtau
                    order2[id] = (unsigned short)(kl << 5 | o);
#pragma unroll
                    for (int c = 0; c < CH; ++c) {
                        if (c >= nc) break;
                        T v[kRec];
#pragma unroll
                        for (int q = 0; q < 11; ++q) v[q] = acc[c][q];
                        v[11] = Lnu[c] * sgd; v[12] = v[13] = v[15] = T(0);
                        v[14] = ((act >> c) & 1u) ? T(1) : T(0);
                        put16<kRec>(rec + id * REC + c * kRec, v);
                    }
                }
                __syncthreads();
                // the steps of every (frequency, sample) in the place of its coefficients
                for (int i = tid; i < n * nc; i += NT) {
                    const int c = i / n, id = i - c * n;
                    T* rp = rec + id * REC + c * kRec;
                    T v[kRec];
                    get16<kRec>(rp, v);
                    if (v[14] == T(0)) continue;
                    ev[6]++;
                    if (gstate) {
                        const int at = order2[id];
                        const long long g = (((long long)(v0 + c) * job.nframes + f) * N + (kr + (at >> 5) - 1)) * npad + jb + (at & 31);
                        put16<12>(gstate + g * kState + 16, v);
                        job.gact[g] = 1;
                    }
                    T w[kRec];
                    step_record(c_moments, v, v[11], w);
                    put16<kRec>(rp, w);
                }
                __syncthreads();
                // 3. composition: lane = ray, every record once per row
                for (int kl = w0; kl < w1; ++kl) {
                    const unsigned bl = ball[kl];
                    if (!((bl >> lane) & 1u)) continue;
                    const T* rp = rec + (base[kl] + __popc(bl & ((1u << lane) - 1u))) * REC;
#pragma unroll
                    for (int q = 0; q < NTASK; ++q) {
                        const int task = q * W + warp, c = task >> 2, row = task & 3;
                        if (c >= nc) continue;
                        T v[kRec];
                        get16<kRec>(rp + c * kRec, v);
                        if (v[14] == T(0)) continue;
                        if (gstate) {
                            const long long g = (((long long)(v0 + c) * job.nframes + f) * N + (kr + kl - 1)) * npad + jb + lane;
                            put16<4>(gstate + g * kState + 4 * row, pr[q]);
                        }
                        T p1[4], p2[4], p3[4];
                        kvec_t(v + 8, pr[q], p1); kvec_t(v + 8, p1, p2); kvec_t(v + 8, p2, p3);
                        ps[q] += pr[q][0] * v[4] + pr[q][1] * v[5] + pr[q][2] * v[6] + pr[q][3] * v[7];
#pragma unroll
                        for (int s = 0; s < 4; ++s) pr[q][s] = v[0] * pr[q][s] + v[1] * p1[s] + v[2] * p2[s] + v[3] * p3[s];
                    }
                }
                __syncthreads();
                w0 = w1;
            }
        }
        if (live) {
#pragma unroll
            for (int q = 0; q < NTASK; ++q) {
                const int task = q * W + warp, c = task >> 2, row = task & 3;
                if (c >= nc) continue;
                T* o = seg_out + (((long long)((v0 + c) * job.nframes + f) * job.nseg + seg) * job.npix + jb + lane) * 20;
                put16<4>(o + 4 * row, pr[q]);
                o[16 + row] = ps[q];
            }
        }
        if (counters) {
            ev[4] = ev[5] * nc;   // every pair's coefficients at every frequency
            for (int q = 0; q < 7; ++q)
                if (ev[q]) atomicAdd(&counters[q], (unsigned long long)ev[q]);
        }
#pragma unroll
        for (int q = 0; q < 7; ++q) ev[q] = 0;
    }
}

// The first sample of each ray beyond its nmax-th passage through |z| < slab (WindingState, step.jl:379-398),
// N + 1 when there is none.
template <class T>
__global__ void k_wind_stop(PlanView P, long long j0, long long npix, long long npad, const T* __restrict__ stream, int nmax, T slab,
                            int* __restrict__ kstop) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= npix) return;
    const int n = int(P.get(PF_NSAMP, j0 + j));
    T zprev = T(0);
    int wn = 0, stop = n + 1;
    bool inside = false, crossed = false, zset = false;
    for (int k = 1; k <= n; ++k) {
        const T* p = stream + (long long)(k - 1) * SM_COUNT * npad + j;
        if (!(stream_flags(p[SM_FLAGS * npad]) & 8u)) continue;
        const T z = p[SM_R * npad] * p[SM_CTH * npad];
        if (!zset) { zset = true; inside = fabs(z) < slab; }
        else {
            const bool now = fabs(z) < slab, crossing = zprev * z < T(0);
            if (inside || now) {
                crossed = crossed || crossing;
                if (inside && !now) { if (crossed) wn += 1; crossed = false; }
                else if (!inside && now) crossed = crossing;
                inside = now;
            } else if (crossing) {
                wn += 1;
            }
        }
        zprev = z;
        if (wn > nmax) { stop = k; break; }
    }
    kstop[j0 + j] = stop;
}

// Front-to-back composition of a ray's segments and the observed Stokes vector (x nuhat^3); `out` holds
// `nout` rays per combination, this launch's from j0.
template <class T>
__global__ void k_compose(TransportJob job, const double* __restrict__ cnu, const T* __restrict__ seg_out, long long nout, double* __restrict__ out) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long ncombo = (long long)job.nframes * job.nfreq;
    if (q >= job.npix * ncombo) return;
    const long long combo = q / job.npix, j = q % job.npix;
    const T* first = seg_out + ((combo * job.nseg) * job.npix + j) * 20;
    double S[4];
    const T* last = first + (long long)(job.nseg - 1) * job.npix * 20;
    for (int r = 0; r < 4; ++r) S[r] = last[16 + r];
    for (int s = job.nseg - 2; s >= 0; --s) {
        const T* PS = first + (long long)s * job.npix * 20;
        double Sn[4];
        for (int r = 0; r < 4; ++r)
            Sn[r] = PS[16 + r] + PS[4 * r] * S[0] + PS[4 * r + 1] * S[1] + PS[4 * r + 2] * S[2] + PS[4 * r + 3] * S[3];
        for (int r = 0; r < 4; ++r) S[r] = Sn[r];
    }
    const int v = int(combo / job.nframes);
    const double nh = cnu[v] / kNU0, n3 = nh * nh * nh;
    double* o = out + (combo * nout + job.j0 + j) * 4;
    for (int r = 0; r < 4; ++r) o[r] = S[r] * n3;
}

}  // namespace ks
