// ks_reverse.cuh -- the reverse pass of the polarized transport, in FP32 or FP64: the gradient of sum(dstokes * Stokes) in every
// parameter of the thermal splats (the reference's dual sweep, src/Splats/dual_gradient.jl).
//
// The forward pass (k_transport with a gstate) leaves, at every active (sample, ray, frequency), the state P of the
// segment before the sample, the summed coefficients and the step length. k_adj_bounds turns the segments' (P, S)
// into the adjoint w_s at each segment's start and the tail T behind its end. k_reverse takes the forward pass's
// work units (32 rays x one segment x one frame x up to CH frequencies) in runs of samples from the last to the
// first, each phase spread over the block:
//   1. tests: the candidate splats of every active (ray, sample), as the forward pass tested them, as bit masks;
//   2. tails: the step records of the stored coefficients, then one thread per (ray, frequency) takes
//      T <- E + O T back to front and leaves the tail behind every sample;
//   3. steps: w = P^T w_s and the step adjoint of every (frequency, sample), c-bar in place of the record;
//   4. elements: the masks turned into one sample list per splat; a warp takes a splat and runs its samples 32 at a
//      time, so that the splat's row is the same for all lanes, and keeps the splat's sums in registers.
// The element adjoint runs backwards (one pass from c-bar to the splat's parameters, the frequencies meeting in
// seven scalars before the frame), where forward-mode duals took four to five partials through every operation; what
// is linear in a splat's constants (the centre, the quaternion, the field's angles) is left as sums over samples
// and turned into parameter rows once, in FP64. Each splat's sums of a window are formed by one warp in a fixed
// order and every unit has its own block of partial sums, so the gradient is the same bit for bit.
//
// Bound by instruction issue (44% of the issue slots at 12 warps per SM, its registers' limit). 224 x 224 x 896, 64 splats,
// three frequencies: 11.1 ms; the step and element kernels before it took 28.7 ms. Four blocks per SM (128 registers) spill:
// the whole gradient 23.6 ms against 22.5.
#pragma once
#include "ks_gradient.cuh"
#include "ks_transport.cuh"

namespace ks {

// the adjoint at each segment's start and the tail behind its end, per (ray, combination):
// bnd[((combo nseg + s) 8 + q) npix + j], q = 0..3 w, 4..7 T; the seeds of all rays, nseeds per combination
template <class T>
__global__ void k_adj_bounds(TransportJob job, const double* __restrict__ cnu, const T* __restrict__ seg_out, const double* __restrict__ seeds,
                             long long nseeds, T* __restrict__ bnd) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long ncombo = (long long)job.nframes * job.nfreq;
    if (q >= job.npix * ncombo) return;
    const long long combo = q / job.npix, j = q % job.npix;
    const int v = int(combo / job.nframes);
    const double nh = cnu[v] / kNU0, n3 = nh * nh * nh;
    const T* base = seg_out + ((combo * job.nseg) * job.npix + j) * 20;
    T* b = bnd + (combo * job.nseg) * 8 * job.npix + j;
    double w[4];
    for (int s = 0; s < 4; ++s) w[s] = seeds[(combo * nseeds + job.j0 + j) * 4 + s] * n3;
    for (int sg = 0; sg < job.nseg; ++sg) {
        const T* PS = base + (long long)sg * job.npix * 20;
        for (int s = 0; s < 4; ++s) b[((long long)sg * 8 + s) * job.npix] = T(w[s]);
        double wn[4];
        for (int s = 0; s < 4; ++s) wn[s] = PS[s] * w[0] + PS[4 + s] * w[1] + PS[8 + s] * w[2] + PS[12 + s] * w[3];
        for (int s = 0; s < 4; ++s) w[s] = wn[s];
    }
    double T4[4] = {0.0, 0.0, 0.0, 0.0};
    for (int sg = job.nseg - 1; sg >= 0; --sg) {
        const T* PS = base + (long long)sg * job.npix * 20;
        for (int s = 0; s < 4; ++s) b[((long long)sg * 8 + 4 + s) * job.npix] = T(T4[s]);
        double Tn[4];
        for (int r = 0; r < 4; ++r) Tn[r] = PS[16 + r] + PS[4 * r] * T4[0] + PS[4 * r + 1] * T4[1] + PS[4 * r + 2] * T4[2] + PS[4 * r + 3] * T4[3];
        for (int r = 0; r < 4; ++r) T4[r] = Tn[r];
    }
}


// the sums over (sample, splat) pairs
enum PairSum {
    PS_E = 0,        // sum s e_j (3): the centre
    PS_E2 = 3,       // sum s e_j^2 (3): the log widths
    PS_N = 6,        // sum s dr_i e_j (9): the quaternion
    PS_PH = 15,      // sum s dq/dphase
    PS_TT = 16,      // sum s tt
    PS_TT2 = 17,     // sum s tt^2
    PS_PHT = 18,     // sum s dq/dphase (t - t0)
    PS_S = 19,       // sum s: ln n_e
    PS_TE = 20, PS_B = 21,
    PS_BH = 22,      // the field direction (3)
    PS_U = 25,       // the velocity (3)
    PS_COUNT = 28
};

// What the fits give back at one frequency: L = c-bar . c and its derivatives by ln Te, ln B, ln nu, cos theta_B, and
// by cos 2chi and sin 2chi.
template <class T>
struct FitBar { T L, te, b, nu, cb, c2, s2; };

// thermal_row and the screen rotation (transport.jl:265-270) backwards: adds to `o` for one frequency. cb: the
// sample's c-bar (11). df0, dkr: the derivatives of the Bessel ratios by ln Te.
template <class T>
__device__ __forceinline__ void thermal_row_bar(const T* r, T ne, T nu, T st, T ct, T c2c, T s2c, T df0, T dkr, const T* cb, FitBar<T>& o) {
    const T Te = r[RW_TE], nc = r[RW_NUC], f0 = r[RW_F0], kr = r[RW_KR];
    const T inu = hrcp(nu), b = nc * inu;
    constexpr double kWP = kEE * kEE / (3.141592653589793 * kME), kRV = 3.141592653589793 * 2.0 / kCL;
    const T nh = nu * T(1.0 / kNU0), i2 = hrcp(nh * nh);
    const T plb = T(kWP) * ne * inu * inu * b;
    const T gV = cb[10] * nh;
    const T jq = cb[1] * c2c + cb[2] * s2c, aq = cb[5] * c2c + cb[6] * s2c, rq = cb[8] * c2c + cb[9] * s2c;
    if (!(st > T(0))) {
        const T k = T(kRV) * nu * plb * ct * gV;   // rV alone, proportional to nu_c nu^-2 f0 cos theta_B (the screen factor nu)
        o.L += k * f0; o.te += k * df0; o.b += k * f0; o.nu -= k * f0;
        if (ct > T(-1) && ct < T(1)) o.cb += T(kRV) * nu * plb * f0 * gV;
        return;
    }
    // Faraday: rQ = pq jf(x), rV = pv ff(x) cos theta_B
    const T x = Te * hsqrt(T(1414.2135623730951) * st * b);
    const bool lo = x < T(120);
    const T q = lo ? x * T(1.0 / 120) : T(120) * hrcp(x);
    const T q2 = q * q, q4 = q2 * q2, q5 = q4 * q, q10 = q5 * q5, q20 = q10 * q10;
    const T s20 = hrcp(T(1) + q20), sw = lo ? q20 * s20 : s20, sw1 = lo ? s20 : q20 * s20;   // sw1 = 1 - sw
    const T lx = hlog2(x + T(1e-16));
    const T ex = T(0.011) * hexp(x * T(-1.0 / 47.2)), exl = ex * x * T(1.0 / 47.2);
    const T px = T(7.9370052598409974e-01 / 67.44733739010397 * 3.141592653589793 * 1e4) * hexp2(fmin(T(-8.0 / 3) * lx, T(100)));
    const T x1 = hexp2(T(1.035) * lx) * T(1.0 / 4.7), e1 = T(2.011) * hexp(-x1);
    const T x2 = hexp2(T(1.2) * lx) * T(1.0 / 2.73), e2 = hexp(-x2);
    T sh, ch;
    fsincos(x * T(0.5), sh, ch);
    const T ext = ex - px;
    const T jf = e1 - ch * e2 - ex + ext * sw;
    const T jfx = -T(1.035) * x1 * e1 + e2 * (T(0.5) * x * sh + T(1.2) * x2 * ch) + exl + (T(8.0 / 3) * px - exl) * sw + T(20) * ext * sw * sw1;
    const T gq = rq * nh * (T(0.5 * kRV) * nu * plb * b * st * st);
    const T kt = kr + T(6) * Te;
    const T rQ = gq * kt * jf, rQx = gq * kt * jfx;              // c-bar . rQ and its derivative by ln x
    const T y0 = T(1) + T(0.035) * x, ff = T(1) - T(0.11) * hln(y0), ffx = T(-0.11 * 0.035) * x * hrcp(y0);
    const T gv = gV * (T(kRV) * nu * plb);
    const T rV = gv * f0 * ff * ct, rx = rQx + gv * f0 * ffx * ct;
    T L = rQ + rV, te = rx + gq * jf * (dkr + T(6) * Te) + gv * df0 * ff * ct, lb = T(2) * rQ + rV + T(0.5) * rx;
    // rQ nu^-3, rV nu^-2, x nu^-1/2; the screen factor is nu
    T ln = T(-2) * rQ - rV - T(0.5) * rx;
    T lst = T(2) * rQ + T(0.5) * rx, lct = gv * f0 * ff;         // by ln sin theta_B, by cos theta_B
    // emission and absorption: j = p f(X), X = nu / nu_s, the absorptivities j / B_nu
    const T nus = T(1.5) * nc * st * Te * Te + T(1), w = (nus - T(1)) * hrcp(nus);
    const T ls = hlog2(nu * hrcp(nus)) * T(1.0 / 3);
    const T c13 = hexp2(-ls), c23 = c13 * c13, u = T(1.8899 / 3) * hexp2(ls);
    const T e13 = hexp(T(-3) * u);
    constexpr double kJ = kEE * kEE / (2.0 * 1.7320508075688772 * kCL);   // times nu first: 2e-30 n_e underflows in FP32
    const T iT = hrcp(Te), ist = hrcp(st), pj = T(kJ) * nu * ne * iT * iT * e13, pI = pj * T(2.5651);
    const T fI = T(1) + T(1.92) * c13 + T(0.9977) * c23, fIx = T(-1.92 / 3) * c13 - T(0.9977 * 2 / 3) * c23;
    const T fQ = T(1) + T(0.93193) * c13 + T(0.499873) * c23, fQx = T(-0.93193 / 3) * c13 - T(0.499873 * 2 / 3) * c23;
    const T v1 = T(1.81384) * nus * inu, v2 = T(3.42319) * c23, v3 = T(0.0292545) * hexp2(T(-1.5) * ls), v4 = T(2.03773) * c13;
    const T fV = v1 + v2 + v3 + v4, fVx = -v1 - T(2.0 / 3) * v2 - T(0.5) * v3 - T(1.0 / 3) * v4;
    const T pVc = pj * T(4.0 / 3) * iT * ist, pV = pVc * ct;
    const T jI = pI * fI, jQ = pI * fQ, jV = pV * fV;
    constexpr double kY = kHPL / (kME * kCL * kCL), kB = 2.0 * kHPL / (kCL * kCL);
    const T y = T(kY) * nu * iT;
    const T em1 = y < T(2e-3) ? y * (T(1) + y * (T(0.5) + y * (T(1.0 / 6) + y * T(1.0 / 24)))) : expm1(y);
    const T iB = planck_inverse(T(kB * 1e33), nu, em1);
    const T ry = y + y * hrcp(em1);                              // d ln(1 / B) / d ln y
    // the cap (coefficients.jl:264-288): jQ, jV scaled by 0.99 jI / sqrt(jQ^2 + jV^2) where that is below one
    T cap = T(1), qq = T(0), vv = T(0), ip2 = T(0);              // ip2 != 0: capped; jQ / jI, jV / jI, 1 / (their squares' sum)
    if (jI > T(0)) {   // the ratios of the fits, as thermal_row takes them
        const T iI = hrcp(fI);
        qq = fQ * iI; vv = T(4.0 / 3 / 2.5651) * iT * ist * ct * fV * iI;
        const T p2 = qq * qq + vv * vv;
        if (p2 > T(0.9801)) {
            cap = T(0.99) * hrsqrt(p2);
            ip2 = hrcp(p2);
        }
    }
    const T ja = nh * iB;
    const T GI = cb[0] * i2 + cb[4] * ja, GQ = jq * i2 + aq * ja, GV = cb[3] * i2 + cb[7] * ja;
    const T jQc = cap * jQ, jVc = cap * jV;
    const T Lj = (cb[0] * jI + jq * jQc + cb[3] * jVc) * i2, La = (cb[4] * jI + aq * jQc + cb[7] * jVc) * ja;
    const T H = ip2 != T(0) ? GQ * qq + GV * vv : T(0);          // cap = 0.99 jI / sqrt(jQ^2 + jV^2)
    const T hI = GI + cap * H, hQ = cap * (GQ - H * qq * ip2), hV = cap * (GV - H * vv * ip2);
    const T sI = hI * jI, sQ = hQ * jQ, sV = hV * jV, all = sI + sQ + sV;
    const T lX = -u * all + hI * pI * fIx + hQ * pI * fQx + hV * pV * fVx;   // by ln X
    L += Lj + La;
    te += T(-2) * (sI + sQ) - T(3) * sV - T(2) * w * lX - ry * La;
    lb -= w * lX;
    ln += all + lX - T(2) * Lj + La + (ry - T(3)) * La;
    lst -= sV + w * lX;
    lct += hV * pVc * fV;
    o.L += L; o.te += te; o.b += lb; o.nu += ln;
    if (ct > T(-1) && ct < T(1)) o.cb += lct - lst * ct * ist * ist;
    // by the rotation: what multiplies cos 2chi and sin 2chi
    const T rQv = T(0.5 * kRV) * nu * plb * b * st * st * kt * jf * nh, Qj = jQc * i2, Qa = jQc * ja;
    o.c2 += cb[1] * Qj + cb[5] * Qa + cb[8] * rQv;
    o.s2 += cb[2] * Qj + cb[6] * Qa + cb[9] * rQv;
}

// row_frame backwards: from the derivatives by ln(1 / g) (`lg`), cos theta_B, cos 2chi and sin 2chi to the field
// direction (bb) and the velocity (ub), both added to.
template <class T>
__device__ __forceinline__ void row_frame_bar(const SampleFrame<T>& F, const T* r, T alpha, T beta, T a_sin_tho, T lg, T cbb, T c2b, T s2b, T* bb, T* ub) {
    const T u[3] = {r[RW_U1], r[RW_U2], r[RW_U3]}, q = r[RW_GQ], gam = r[RW_GAM];
    const T b[3] = {r[RW_BX], r[RW_BY], r[RW_BZ]};
    const T ud = u[0] * F.pz[1] + u[1] * F.pz[2] + u[2] * F.pz[3];
    const T ig = gam * F.pz[0] - ud, g = hrcp(ig), udq = ud * q - F.pz[0];
    T m[3], k[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) { m[i] = F.pz[i + 1] + u[i] * udq; k[i] = m[i] * g; }
    T f[3] = {k[1] * b[2] - k[2] * b[1], k[2] * b[0] - k[0] * b[2], k[0] * b[1] - k[1] * b[0]};
    const T fn2 = f[0] * f[0] + f[1] * f[1] + f[2] * f[2];
    T kb[3] = {b[0] * cbb, b[1] * cbb, b[2] * cbb};
    T du[3] = {T(0), T(0), T(0)}, db[3] = {k[0] * cbb, k[1] * cbb, k[2] * cbb}, qb = T(0);
    if (fn2 > T(0)) {
        const T fi = hrsqrt(fn2);
#pragma unroll
        for (int i = 0; i < 3; ++i) f[i] *= fi;
        const T fd = u[0] * f[0] + u[1] * f[1] + u[2] * f[2], fdq = fd * q;
        const T fz1 = f[0] + u[0] * fdq, fz2 = f[1] + u[1] * fdq, fz3 = f[2] + u[2] * fdq;
        const T ft = F.lapse_inv * fd, fr = F.sDS * fz1, fth = F.misS * fz3, fph = F.om_lapse * fd + F.ivarpi * fz2;
        const T a = F.a, rr = F.r, s = F.sth, c = F.cth, as2 = a * s * s, ra = rr * rr + a * a;
        const T Aw = F.pu[0] * fr - F.pu[1] * ft + as2 * (F.pu[1] * fph - F.pu[3] * fr);
        const T Bw = (ra * (F.pu[3] * fth - F.pu[2] * fph) - a * (F.pu[0] * fth - F.pu[2] * ft)) * s;
        const T k1 = Aw * rr - Bw * a * c, k2 = -(Aw * a * c + Bw * rr);
        const T mu = -(alpha + a_sin_tho), y = mu * k1 - beta * k2, x = beta * k1 + mu * k2, r2 = x * x + y * y;
        if (r2 > T(0)) {
            const T ir = hrcp(r2);
            // d chi = (x dy - y dx) / r2; cos 2chi = (x^2 - y^2) / r2, sin 2chi = 2 x y / r2
            const T chi = T(2) * ((x * x - y * y) * s2b - T(2) * x * y * c2b) * ir * ir;
            const T xb = -chi * y, yb = chi * x;
            const T k1b = mu * yb + beta * xb, k2b = mu * xb - beta * yb;
            const T Ab = rr * k1b - a * c * k2b, Bb = (-a * c * k1b - rr * k2b) * s;
            const T frb = Ab * (F.pu[0] - as2 * F.pu[3]), ftb = Bb * a * F.pu[2] - Ab * F.pu[1];
            const T fphb = Ab * as2 * F.pu[1] - Bb * ra * F.pu[2], fthb = Bb * (ra * F.pu[3] - a * F.pu[0]);
            const T z[3] = {F.sDS * frb, F.ivarpi * fphb, F.misS * fthb};
            const T fdqb = u[0] * z[0] + u[1] * z[1] + u[2] * z[2];
            const T fdb = F.lapse_inv * ftb + F.om_lapse * fphb + q * fdqb;
            qb += fd * fdqb;
            // chi does not change with the length of f, so the normalisation passes f-bar through (times 1 / |f|)
            T fb[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                du[i] += fdq * z[i] + fdb * f[i];
                fb[i] = fi * (z[i] + u[i] * fdb);
            }
            kb[0] += b[1] * fb[2] - b[2] * fb[1]; kb[1] += b[2] * fb[0] - b[0] * fb[2]; kb[2] += b[0] * fb[1] - b[1] * fb[0];
            db[0] += fb[1] * k[2] - fb[2] * k[1]; db[1] += fb[2] * k[0] - fb[0] * k[2]; db[2] += fb[0] * k[1] - fb[1] * k[0];
        }
    }
    const T gb = kb[0] * m[0] + kb[1] * m[1] + kb[2] * m[2];
    const T udqb = (kb[0] * u[0] + kb[1] * u[1] + kb[2] * u[2]) * g;
    const T igb = (lg - gb * g) * g;                              // lg / ig - gb / ig^2
    const T udb = q * udqb - igb;
    qb += ud * udqb;
    const T gamb = (igb * F.pz[0] - qb * q * q) * hrcp(gam);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        ub[i] += du[i] + kb[i] * g * udq + udb * F.pz[i + 1] + gamb * u[i];
        bb[i] += db[i];
    }
}

// The sums of one (sample, splat) pair, added to v. sample: its position, emission time, frame; cbs: its records
// (c-bar per frequency, kRec apart, the active flag at 14).
template <class T>
__device__ __forceinline__ void pair_adjoint(const T* r, T x, T y, T z, T t, const SampleFrame<T>& F, T alpha, T beta, T a_sin_tho, const T* nu, int nc,
                                             const T* cbs, T* v) {
    const T dt = t - r[RW_T0];
    T sp, cp;
    sincos_product(r[RW_OMEGA], dt, sp, cp);
    const T cx = r[RW_CX], cy = r[RW_CY];
    const T d0 = x - (cx * cp - cy * sp), d1 = y - (cx * sp + cy * cp);
    const T dr[3] = {d0 * cp + d1 * sp, -d0 * sp + d1 * cp, z - r[RW_CZ]};
    T e[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) e[j] = r[RW_A0 + j] * dr[0] + r[RW_A3 + j] * dr[1] + r[RW_A6 + j] * dr[2];
    const T tt = dt * r[RW_INVW];
    const T ne = r[RW_NE] * weight_of((e[0] * e[0] + e[1] * e[1] + e[2] * e[2] + tt * tt) * T(0.5));
    const LFrame<T> lf = row_frame(F, r, alpha, beta, a_sin_tho);
    T sb, cb;
    pitch_sc(lf.cosB, sb, cb);
    FitBar<T> o{T(0), T(0), T(0), T(0), T(0), T(0), T(0)};
    const T df0 = r[RW_DF0], dkr = r[RW_DKR];
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
        T w[kRec];
        get16<kRec>(cbs + c * kRec, w);
        if (w[14] == T(0)) continue;
        thermal_row_bar(r, ne, nu[c] * lf.g, sb, cb, lf.c2c, lf.s2c, df0, dkr, w, o);
    }
    row_frame_bar(F, r, alpha, beta, a_sin_tho, o.nu, o.cb, o.c2, o.s2, v + PS_BH, v + PS_U);
    const T s = o.L;
    const T g0 = r[RW_A0] * e[0] + r[RW_A1] * e[1] + r[RW_A2] * e[2], g1 = r[RW_A3] * e[0] + r[RW_A4] * e[1] + r[RW_A5] * e[2];
    const T ph = s * (g0 * (dr[1] + cy) - g1 * (dr[0] + cx));
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const T se = s * e[j];
        v[PS_E + j] += se;
        v[PS_E2 + j] += se * e[j];
#pragma unroll
        for (int i = 0; i < 3; ++i) v[PS_N + 3 * i + j] += se * dr[i];
    }
    v[PS_PH] += ph; v[PS_TT] += s * tt; v[PS_TT2] += s * tt * tt; v[PS_PHT] += ph * dt; v[PS_S] += s;
    v[PS_TE] += o.te; v[PS_B] += o.b;
}

// The sum over the warp of each of 32 values, value l in lane l: five steps that halve the values and fold the lanes.
template <class T>
__device__ __forceinline__ T warp_sums(T v[32], int lane) {
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int q = 0; q < h; ++q) {
            const T keep = up ? v[q + h] : v[q], give = up ? v[q] : v[q + h];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
    return v[0];
}

// the place of the n-th (from 0) set bit of m
__device__ __forceinline__ int nth_bit(unsigned m, int n) {
    int p = 0;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const int c = __popc(m & ((1u << h) - 1u));
        if (n >= c) { n -= c; m >>= h; p += h; }
    }
    return p;
}

template <class T, int CH, int NT>
struct ReverseSmem {
    static constexpr int W = NT / 32, ST = row_stride<T, 1>(), REC = CH * kRec + 16 / int(sizeof(T));
    __host__ __device__ static size_t rows_bytes(int ntot) { return (size_t(ntot) * ST * sizeof(T) + 15) / 16 * 16; }
    __host__ __device__ static size_t bytes(int ntot, int run, int cap, bool rows_shared) {
        const int nw = (ntot + 31) / 32;
        return (rows_shared ? rows_bytes(ntot) : 0) + (size_t(cap) * REC + 5 * 32 + CH * 4 * 32 + CH + 4) * sizeof(T)              // rows, records, rays, w
               + size_t(run) * 32 * nw * 4 + size_t(nw) * W * 4 + size_t(ntot) * (cap / 32) * 4                            // masks, candidates, lists
               + W * 10 * 4 + run * 8 + size_t(run) * 32 + size_t(cap) * 2 + size_t(ntot) * 2 + 64;                        // boxes, lane masks, flags, orders
    }
};

template <class T, int CH, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
k_reverse(PlanView P, Spacetime st, TransportJob job, const T* __restrict__ rows_g, const double* __restrict__ ct, const double* __restrict__ cnu,
          const T* __restrict__ stream, const T* __restrict__ bnd, unsigned long long* __restrict__ work, T* __restrict__ gunit,
          unsigned* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem[];
    using SM = ReverseSmem<T, CH, NT>;
    constexpr int W = NT / 32, ST = SM::ST, REC = SM::REC;
    static_assert(W >= CH, "a warp per frequency takes the tails");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntot = job.ntot, nw = (ntot + 31) >> 5, R = job.run, RS = R / W, cap = job.cap, TW = cap >> 5;
    unsigned char* smem_at = smem;
    const T* rows = rows_g;
    if (job.rows_shared) {
        __shared__ __align__(8) unsigned long long bar;
        const unsigned bytes = unsigned(SM::rows_bytes(ntot));
        if (bytes > 0 && !stage_bulk(smem, rows_g, bytes, &bar, job.stage_test == 0, job.stage_test ? 4096 : kStageWaitLimit)) {
            if (tid == 0) atomicOr(err, 1u);
            return;
        }
        rows = reinterpret_cast<const T*>(smem);
        smem_at += bytes;
    }
    T* rec = reinterpret_cast<T*>(smem_at);                             // [cap][REC]
    T* rayc = rec + (long long)cap * REC;                               // [5][32]
    T* ws = rayc + 5 * 32;                                              // [CH][4][32]: w at the segment's start
    T* nu = ws + CH * 4 * 32;                                           // [CH] (+ 4)
    unsigned* masks = reinterpret_cast<unsigned*>(nu + CH + 4);         // [run][nw][32]
    unsigned* cand = masks + R * nw * 32;                               // [W][nw]
    unsigned* lists = cand + W * nw;                                    // [ntot][TW]: the records each splat reaches
    float* boxes = reinterpret_cast<float*>(lists + ntot * TW);         // [W][10]
    unsigned* ball = reinterpret_cast<unsigned*>(boxes + W * 10);       // [run]: the active rays
    int* base = reinterpret_cast<int*>(ball + R);                       // [run]
    unsigned char* actb = reinterpret_cast<unsigned char*>(base + R);   // [run][32]: the active frequencies
    unsigned short* order = reinterpret_cast<unsigned short*>(actb + R * 32);   // [cap]: sample << 5 | lane of a record
    unsigned short* livel = order + cap;                                // [ntot]: the window's splats
    __shared__ unsigned long long s_unit;
    __shared__ int s_live, s_next;
    const T a = T(st.a), a_sin_tho = T(st.a * sin(st.thetao));
    const T* gstate = static_cast<const T*>(job.gstate);
    const int N = st.N;
    const long long npad = job.npad, fs = npad, gsz = (long long)ntot * PS_COUNT;
    const int per_chunk = job.nseg * job.nframes * job.nvc;
    const long long total = job.nchunks * per_chunk;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_unit = atomicAdd(work, 1ull);
        __syncthreads();
        if (s_unit >= (unsigned long long)total) break;
        const long long u = total - 1 - (long long)s_unit;
        const long long jb = u / per_chunk * 32;
        const int rem = int(u % per_chunk), seg = rem / (job.nframes * job.nvc), y = rem % (job.nframes * job.nvc);
        const int f = y / job.nvc, v0 = (y % job.nvc) * CH, nc = min(CH, job.nfreq - v0);
        const bool live = jb + lane < job.npix;
        const long long jl = live ? jb + lane : job.npix - 1, jp = job.j0 + jl;   // in the stream, in the plan
        const int k0 = 1 + seg * job.seg_len;
        int klim = live ? int(P.get(PF_NSAMP, jp)) : 0;
        if (job.kstop && live) klim = min(klim, job.kstop[jp] - 1);
        const int k1 = min(k0 + job.seg_len, __reduce_max_sync(0xffffffffu, klim) + 1);
        if (warp == 0) {
            rayc[lane] = T(P.get(PF_ALPHA, jp)); rayc[32 + lane] = T(P.get(PF_BETA, jp)); rayc[64 + lane] = T(P.get(PF_ETA, jp));
            rayc[96 + lane] = T(P.get(PF_LAM, jp)); rayc[128 + lane] = T(P.get(PF_DTAU, jp));
        }
        if (tid < nc) nu[tid] = T(cnu[v0 + tid]);
        T* gu = gunit + u * gsz;
        for (long long q = tid; q < gsz; q += NT) gu[q] = T(0);
        // warp c < nc carries the tails of frequency c
        T T4[4] = {T(0), T(0), T(0), T(0)};
        if (warp < nc) {
            const long long combo = (long long)(v0 + warp) * job.nframes + f;
            const T* b = bnd + (combo * job.nseg + seg) * 8 * job.npix + jl;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ws[(warp * 4 + q) * 32 + lane] = live ? b[(long long)q * job.npix] : T(0);
                T4[q] = live ? b[(long long)(4 + q) * job.npix] : T(0);
            }
        }
        const T t_obs = T(ct[f]);
        if (k1 <= k0) continue;
        for (int kr = k0 + (k1 - 1 - k0) / R * R; kr >= k0; kr -= R) {
            const T* sp = stream + (long long)(kr - 1) * SM_COUNT * npad + jl;
            __syncthreads();   // the last window's scan of `ball` is over
            // 1. the active samples, their candidates, the tests
            {
                UnitBox b = unit_box_empty();
                for (int s = 0; s < RS; ++s) {
                    const int kl = warp * RS + s;
                    unsigned act = 0u;
                    if (kr + kl <= klim && kr + kl < k1)
                        for (int c = 0; c < nc; ++c)
                            act |= unsigned(job.gact[(((long long)(v0 + c) * job.nframes + f) * N + (kr + kl - 1)) * npad + jl]) << c;
                    actb[kl * 32 + lane] = (unsigned char)act;
                    const unsigned bl = __ballot_sync(0xffffffffu, act != 0u);
                    if (lane == 0) ball[kl] = bl;
                    if (act) {
                        const T* p = sp + (long long)kl * SM_COUNT * fs;
                        unit_box_add(b, float(p[SM_X * fs]), float(p[SM_Y * fs]), float(p[SM_Z * fs]), float(p[SM_T * fs]));
                    }
                }
                unit_box_reduce(b);
                const float* bf = reinterpret_cast<const float*>(&b);
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 10; ++q) boxes[warp * 10 + q] = bf[q];
            }
            __syncthreads();
            const int G = max(1, min(W, 16 / RS)), g0 = warp / G * G;
            {
                UnitBox b = unit_box_empty();
                for (int q = g0; q < g0 + G; ++q) {
                    const float* o = boxes + q * 10;
                    b.xlo = fminf(b.xlo, o[0]); b.xhi = fmaxf(b.xhi, o[1]); b.ylo = fminf(b.ylo, o[2]); b.yhi = fmaxf(b.yhi, o[3]);
                    b.zlo = fminf(b.zlo, o[4]); b.zhi = fmaxf(b.zhi, o[5]); b.rlo = fminf(b.rlo, o[6]); b.rhi = fmaxf(b.rhi, o[7]);
                    b.slo = fminf(b.slo, o[8]); b.shi = fmaxf(b.shi, o[9]);
                }
                for (int wd = warp - g0; wd < nw; wd += G) {
                    const int i = wd * 32 + lane;
                    const unsigned m = __ballot_sync(0xffffffffu, i < ntot && b.xlo <= b.xhi && row_reaches(rows + (long long)i * ST, b, t_obs));
                    if (lane == 0) cand[g0 / G * nw + wd] = m;
                }
            }
            __syncthreads();
            for (int s = 0; s < RS; ++s) {
                const int kl = warp * RS + s;
                if (ball[kl] == 0u) continue;
                const bool test = (ball[kl] >> lane) & 1u;
                const T* p = sp + (long long)kl * SM_COUNT * fs;
                T x = T(0), yy = T(0), z = T(0), t = T(0), rho = T(0);
                if (test) { x = p[SM_X * fs]; yy = p[SM_Y * fs]; z = p[SM_Z * fs]; t = t_obs - p[SM_T * fs]; rho = sqrt(x * x + yy * yy); }
                for (int wd = 0; wd < nw; ++wd) {
                    unsigned m = 0u, c = cand[warp / G * nw + wd];
                    while (c) {
                        const int b = __ffs(c) - 1;
                        c &= c - 1;
                        const T* r = rows + (long long)(wd * 32 + b) * ST;
                        if (!test) continue;
                        const T dr = rho - r[RW_RHO], dz = z - r[RW_CZ];
                        if (dr * dr + dz * dz > r[RW_SUPP]) continue;
                        T q;
                        if (!row_exponent<true>(r, t, x, yy, z, q)) continue;
                        if (q < T(kQCUT)) m |= 1u << b;
                    }
                    masks[(kl * nw + wd) * 32 + lane] = m;
                }
            }
            __syncthreads();
            // windows of whole samples whose records fit, the last first
            for (int w1 = R; w1 > 0;) {
                int w0 = w1, n = 0;
                for (; w0 > 0; --w0) {
                    const int c = __popc(ball[w0 - 1]);
                    if (n + c > cap) break;
                    n += c;
                }
                if (n == 0) { w1 = w0; continue; }
                if (tid == 0) {
                    int o = 0;
                    for (int kl = w0; kl < w1; ++kl) { base[kl] = o; o += __popc(ball[kl]); }
                    s_live = 0; s_next = 0;
                }
                for (int q = tid; q < ntot * TW; q += NT) lists[q] = 0u;
                __syncthreads();
                for (int kl = w0 + warp; kl < w1; kl += W) {
                    if (!((ball[kl] >> lane) & 1u)) continue;
                    const int id = base[kl] + __popc(ball[kl] & ((1u << lane) - 1u));
                    order[id] = (unsigned short)(kl << 5 | lane);
                    for (int wd = 0; wd < nw; ++wd) {
                        unsigned m = masks[(kl * nw + wd) * 32 + lane];
                        while (m) {
                            const int b = __ffs(m) - 1;
                            m &= m - 1;
                            atomicOr(&lists[(wd * 32 + b) * TW + (id >> 5)], 1u << (id & 31));
                        }
                    }
                }
                __syncthreads();
                // 2. the step records of the stored coefficients
                for (int i = tid; i < n * nc; i += NT) {
                    const int c = i / n, id = i - c * n, at = order[id];
                    T* rp = rec + id * REC + c * kRec;
                    if (!((actb[at] >> c) & 1u)) { rp[14] = T(0); continue; }
                    const long long g = (((long long)(v0 + c) * job.nframes + f) * N + (kr + (at >> 5) - 1)) * npad + jb + (at & 31);
                    T v[kRec], w[kRec];
                    get16<12>(gstate + g * kState + 16, v);
                    step_record(c_moments, v, v[11], w);
                    put16<kRec>(rp, w);
                }
                // the splats with a sample in the window
                for (int i = tid; i < ntot; i += NT) {
                    unsigned any = 0u;
                    for (int q = 0; q < TW; ++q) any |= lists[i * TW + q];
                    if (any) livel[atomicAdd(&s_live, 1)] = (unsigned short)i;
                }
                __syncthreads();
                // the tails behind the samples, in the place of E
                if (warp < nc) {
                    for (int kl = w1 - 1; kl >= w0; --kl) {
                        const unsigned bl = ball[kl];
                        if (!((bl >> lane) & 1u)) continue;
                        T* rp = rec + (base[kl] + __popc(bl & ((1u << lane) - 1u))) * REC + warp * kRec;
                        T v[kRec];
                        get16<kRec>(rp, v);
                        if (v[14] == T(0)) continue;
                        put16<4>(rp + 4, T4);
                        T t1[4], t2[4], t3[4];
                        kvec(v + 8, T4, t1); kvec(v + 8, t1, t2); kvec(v + 8, t2, t3);
#pragma unroll
                        for (int q = 0; q < 4; ++q) T4[q] = v[4 + q] + v[0] * T4[q] + v[1] * t1[q] + v[2] * t2[q] + v[3] * t3[q];
                    }
                }
                __syncthreads();
                // 3. the step adjoints: c-bar
                for (int i = tid; i < n * nc; i += NT) {
                    const int c = i / n, id = i - c * n, at = order[id], o = at & 31;
                    T* rp = rec + id * REC + c * kRec;
                    if (rp[14] == T(0)) continue;
                    const long long g = (((long long)(v0 + c) * job.nframes + f) * N + (kr + (at >> 5) - 1)) * npad + jb + o;
                    T Pm[16], in[12], wk[4], Rt[4], O[16], E[4], cb[12];
                    get16<16>(gstate + g * kState, Pm);
                    get16<12>(gstate + g * kState + 16, in);
                    get16<4>(rp + 4, Rt);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        wk[q] = Pm[q] * ws[(c * 4) * 32 + o] + Pm[4 + q] * ws[(c * 4 + 1) * 32 + o] + Pm[8 + q] * ws[(c * 4 + 2) * 32 + o] +
                                Pm[12 + q] * ws[(c * 4 + 3) * 32 + o];
                    sample_adjoint_structured(c_moments, in, in[11], wk, Rt, O, E, cb);
                    cb[11] = T(0);
                    put16<12>(rp, cb);
                }
                __syncthreads();
                // 4. the elements: a warp takes a splat
                const int nlive = s_live;
                for (;;) {
                    int li = 0;
                    if (lane == 0) li = atomicAdd(&s_next, 1);
                    li = __shfl_sync(0xffffffffu, li, 0);
                    if (li >= nlive) break;
                    const int i = livel[li];
                    const T* r = rows + (long long)i * ST;
                    const unsigned* lw = lists + i * TW;
                    int cnt = 0;
                    for (int q = 0; q < TW; ++q) cnt += __popc(lw[q]);
                    T v[32];
#pragma unroll
                    for (int q = 0; q < 32; ++q) v[q] = T(0);
                    for (int at0 = 0; at0 < cnt; at0 += 32) {
                        int n0 = at0 + lane;
                        if (n0 >= cnt) continue;
                        int wd = 0;
                        for (; wd < TW; ++wd) {
                            const int c = __popc(lw[wd]);
                            if (n0 < c) break;
                            n0 -= c;
                        }
                        const int id = wd * 32 + nth_bit(lw[wd], n0), at = order[id], o = at & 31;
                        const T* p = stream + (long long)(kr + (at >> 5) - 1) * SM_COUNT * npad + jb + o;
                        const unsigned fl = stream_flags(p[SM_FLAGS * fs]);
                        const SampleFrame<T> F = sample_frame(a, p[SM_R * fs], T(0), p[SM_STH * fs], p[SM_CTH * fs], rayc[64 + o], rayc[96 + o],
                                                                  (fl & 2u) != 0u, (fl & 4u) != 0u);
                        pair_adjoint(r, p[SM_X * fs], p[SM_Y * fs], p[SM_Z * fs], t_obs - p[SM_T * fs], F, rayc[o], rayc[32 + o], a_sin_tho, nu, nc,
                                         rec + id * REC, v);
                    }
                    __syncwarp();
                    const T sum = warp_sums(v, lane);
                    if (lane < PS_COUNT) gu[(long long)i * PS_COUNT + lane] += sum;
                }
                __syncthreads();
                w1 = w0;
            }
        }
    }
}

// The sum over work units in a fixed order: the units of each chunk, one thread per entry and chunk.
template <class T>
__global__ void k_unit_reduce1(const T* __restrict__ gunit, long long nunits, long long gsz, int per_chunk, double* __restrict__ part) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= gsz) return;
    const long long u0 = (long long)blockIdx.y * per_chunk, u1 = min(nunits, u0 + per_chunk);
    double s = 0.0;
    for (long long uu = u0; uu < u1; ++uu) s += gunit[uu * gsz + e];
    part[(long long)blockIdx.y * gsz + e] = s;
}

// The unit sums (added per chunk by k_unit_reduce1) over the chunks in a fixed order, and the 21 parameter rows of
// each splat from its sums.
static __global__ void k_reverse_rows(const double* __restrict__ part, int nchunks, int ntot, const double* __restrict__ tab, const double* __restrict__ gtab,
                               int add, double* __restrict__ out) {
    const int i = blockIdx.x;
    __shared__ double s[PS_COUNT];
    if (threadIdx.x < PS_COUNT) {
        double a = 0.0;
        for (int ch = 0; ch < nchunks; ++ch) a += part[((long long)ch * ntot + i) * PS_COUNT + threadIdx.x];
        s[threadIdx.x] = a;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double* p = tab + (long long)i * ST_COUNT;
    const double* gt = gtab + (long long)i * GT_COUNT;
    double g[GR_COUNT];
    const double es[3] = {p[ST_ES1], p[ST_ES2], p[ST_ES3]};
    for (int k = 0; k < 3; ++k) {
        g[GR_X + k] = p[ST_R0 + 3 * k] * es[0] * s[PS_E] + p[ST_R0 + 3 * k + 1] * es[1] * s[PS_E + 1] + p[ST_R0 + 3 * k + 2] * es[2] * s[PS_E + 2];
        g[GR_S1 + k] = s[PS_E2 + k];
        g[GR_U1 + k] = s[PS_U + k];
    }
    double GM[9];
    for (int q = 0; q < 9; ++q) GM[q] = s[PS_N + q] * es[q % 3];
    const double w = gt[GT_QW], qx = gt[GT_QX], qy = gt[GT_QY], qz = gt[GT_QZ], in = 1.0 / gt[GT_QN];
    double gq[4];
    gq[0] = 2.0 * (-qz * GM[1] + qy * GM[2] + qz * GM[3] - qx * GM[5] - qy * GM[6] + qx * GM[7]);
    gq[1] = 2.0 * (qy * GM[1] + qz * GM[2] + qy * GM[3] - 2.0 * qx * GM[4] - w * GM[5] + qz * GM[6] + w * GM[7] - 2.0 * qx * GM[8]);
    gq[2] = 2.0 * (-2.0 * qy * GM[0] + qx * GM[1] + w * GM[2] + qx * GM[3] + qz * GM[5] - w * GM[6] + qz * GM[7] - 2.0 * qy * GM[8]);
    gq[3] = 2.0 * (-2.0 * qz * GM[0] - w * GM[1] + qx * GM[2] + w * GM[3] - 2.0 * qz * GM[4] + qy * GM[5] + qx * GM[6] + qy * GM[7]);
    const double dot = w * gq[0] + qx * gq[1] + qy * gq[2] + qz * gq[3];
    g[GR_Q1] = -(gq[0] - w * dot) * in;
    g[GR_Q2] = -(gq[1] - qx * dot) * in;
    g[GR_Q3] = -(gq[2] - qy * dot) * in;
    g[GR_Q4] = -(gq[3] - qz * dot) * in;
    g[GR_T0] = p[ST_OMEGA] * s[PS_PH] + p[ST_INVW] * s[PS_TT];
    g[GR_LOGW] = s[PS_TT2];
    g[GR_OMEGA] = -s[PS_PHT];
    g[GR_LOGNE] = s[PS_S];
    g[GR_LOGTE] = s[PS_TE];
    g[GR_LOGB] = s[PS_B];
    const bool field = p[ST_BZERO] == 0.0;
    g[GR_THB] = field ? gt[GT_DBT0] * s[PS_BH] + gt[GT_DBT1] * s[PS_BH + 1] + gt[GT_DBT2] * s[PS_BH + 2] : 0.0;
    g[GR_PHB] = field ? gt[GT_DBP0] * s[PS_BH] + gt[GT_DBP1] * s[PS_BH + 1] + gt[GT_DBP2] * s[PS_BH + 2] : 0.0;
    double* o = out + (long long)i * GR_COUNT;
    for (int q = 0; q < GR_COUNT; ++q) o[q] = add ? o[q] + g[q] : g[q];
}

}  // namespace ks
