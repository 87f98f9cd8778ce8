// ks_adjoint.cuh -- the adjoint of the polarized transport with respect to the splat parameters
// (the reference's dual sweep, src/Splats/dual_gradient.jl, for PolarizedSplats).
//
// Along a ray the observed invariant Stokes vector is the tail T_1 of T_k = E_k + O_k T_{k+1}
// (T_{N+1} = 0); for l = w_1 . T_1 the adjoint in front of sample k is w_k = O_{k-1}^T ... O_1^T w_1
// and the sample's step enters l through w_k^T (O_k T_{k+1} + Ej_k j_k). So
//   j-bar = Ej^T w exactly (E is linear in j), and (alpha-bar, rho-bar) are the partials of
//   w^T (O T + Ej j) by seven forward-mode duals through the step operator (sample_adjoint,
//   transport.jl:221-245);
//   each splat's coefficients c_i enter through c-bar . c_i (ks_reverse.cuh).
// Samples that the forward pass skips (invalid, inside r_h (1 + 1e-3), beyond the half-orbit cutoff,
// or with no active element) have O = 1, E = 0 and no adjoint; culled splats and weights below the
// cutoff contribute nothing, as in the reference.
//
// Here: the gradient's per-splat constants, chi^2 and its seeds, J v and the normal matrix.
#pragma once
#include "ks_gradient.cuh"

namespace {

using namespace ks;

// Per-splat constants of the gradient of THERMAL21 splats: d(K0/K2)/d(logTe), d(K1/K2)/d(logTe) at
// x = 1/Theta_e (dK0/dx = -K1, dK1/dx = -K0 - K1/x), the derivatives of the field direction by its
// angles, and the normalised quaternion with its norm.
__global__ void k_grad_table(int nsplat, int first, const double* __restrict__ params, double* __restrict__ gtab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nsplat) return;
    const double* p = params + 21LL * i;
    double* o = gtab + (long long)(first + i) * GT_COUNT;
    const double Te = exp(p[13]);
    const double xb = 1.0 / Te;
    double k0, k1;
    besselk01(xb, k0, k1);
    const double k2 = k0 + 2.0 * k1 / xb;
    if (k2 > 0) {
        const double dk0 = -k1, dk1 = -k0 - k1 / xb;
        const double dk2 = dk0 + 2.0 * dk1 / xb - 2.0 * k1 / (xb * xb);
        const double df0dx = (dk0 * k2 - k0 * dk2) / (k2 * k2), dkrdx = (dk1 * k2 - k1 * dk2) / (k2 * k2);
        o[GT_DF0] = -xb * df0dx;   // dx/dlogTe = -x
        o[GT_DKR] = -xb * dkrdx;
    } else {
        o[GT_DF0] = 0.0; o[GT_DKR] = 0.0;
    }
    const double st = sin(p[15]), ct = cos(p[15]), sp = sin(p[16]), cp = cos(p[16]);
    o[GT_DBT0] = ct * cp; o[GT_DBT1] = ct * sp; o[GT_DBT2] = -st;
    o[GT_DBP0] = -st * sp; o[GT_DBP1] = st * cp; o[GT_DBP2] = 0.0;
    const double n = sqrt(p[6] * p[6] + p[7] * p[7] + p[8] * p[8] + p[9] * p[9]);
    o[GT_QW] = p[6] / n; o[GT_QX] = p[7] / n; o[GT_QY] = p[8] / n; o[GT_QZ] = p[9] / n; o[GT_QN] = n;
}

// sample_adjoint of n independent samples (FP64): method 0 the structured partials, 1 the seven duals
// through the step operator; out[31 i ..] = O (16), E (4), c-bar (11)
__global__ void k_sample_adjoint(long long n, const double* __restrict__ in, const double* __restrict__ Dl, const double* __restrict__ w,
                                 const double* __restrict__ R, int method, double* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double O[16], E[4], cb[11];
    if (method == 0) sample_adjoint_structured(c_moments, in + 11 * i, Dl[i], w + 4 * i, R + 4 * i, O, E, cb);
    else sample_adjoint(c_moments, in + 11 * i, Dl[i], w + 4 * i, R + 4 * i, O, E, cb);
    double* o = out + 31 * i;
    for (int q = 0; q < 16; ++q) o[q] = O[q];
    for (int q = 0; q < 4; ++q) o[16 + q] = E[q];
    for (int q = 0; q < 11; ++q) o[20 + q] = cb[q];
}

// Image-domain chi^2 and its seed (_frame_seed!, src/Fit/Fit.jl:537-577): for every sorted ray j and
// combination c, r = (image - data) / sigma with data, sigma and mask in screen order; chi^2 = sum r^2
// over unmasked pixels and Stokes, seed = 2 r / sigma (zero where masked). Per-block partial sums.
__global__ void k_chi2_seed(const double* __restrict__ img, const long long* __restrict__ perm, long long npix, int ncombo,
                            const double* __restrict__ data, const double* __restrict__ sigma, double sigma_s,
                            const unsigned char* __restrict__ mask, double* __restrict__ seed, double* __restrict__ partial) {
    __shared__ double sh[256];
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    double acc = 0.0;
    if (idx < npix * ncombo) {
        const long long j = idx % npix, c = idx / npix;
        const long long scr = c * npix + perm[j];
        const bool use = mask ? mask[scr] != 0 : true;
        for (int s = 0; s < 4; ++s) {
            double sd = 0.0;
            if (use) {
                const double sg = sigma ? sigma[scr * 4 + s] : sigma_s;
                const double r = (img[idx * 4 + s] - data[scr * 4 + s]) / sg;
                acc += r * r;
                sd = 2.0 * r / sg;
            }
            seed[idx * 4 + s] = sd;
        }
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// sum of n partials in a fixed order (one block)
__global__ void k_sum_partials(const double* __restrict__ partial, long long n, double* __restrict__ out) {
    __shared__ double sh[256];
    double s = 0.0;
    for (long long q = threadIdx.x; q < n; q += blockDim.x) s += partial[q];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sh[0];
}

// screen- or sorted-order adjoint seeds (ks_adjoint's dstokes) into sorted order
__global__ void k_sort_seed(const double* __restrict__ src, const long long* __restrict__ perm, long long npix, int ncombo, int screen,
                            double* __restrict__ dst) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= npix * ncombo) return;
    const long long j = idx % npix, c = idx / npix;
    const long long sidx = screen ? c * npix + perm[j] : idx;
    for (int s = 0; s < 4; ++s) dst[idx * 4 + s] = src[sidx * 4 + s];
}

}  // namespace

namespace {

using namespace ks;

}  // namespace

// ---- forward mode: J v of the image (jvp!, src/Fit/gauss_newton.jl:91-118) ---------------------------
//
// The reference runs its tails pass on parameters that carry duals along v. Here the splat table of the
// THERMAL21 splats is built as duals (each entry with its K directional derivatives), the march stays
// plain (the geodesics do not depend on the splats), and the consumer composes (P, S) on duals: the
// weight, the frame, the thermal fits, the cap, the invariants, the rotation and the exact step are
// the same templates as the forward path, instantiated on Dual<S, K>.

namespace {

using namespace ks;

// One THERMAL21 column and K tangent directions v[k * 21 + row] -> the dual table row. The cull radii
// (ST_SUPP, ST_RHO) keep their values: the cull is a threshold, not a function of the parameters.
template <class S, int K>
__global__ void k_dual_table(int nsplat, const double* __restrict__ params, const double* __restrict__ dirs, long long dir_stride,
                             const double* __restrict__ tab, const double* __restrict__ gtab, Dual<S, K>* __restrict__ dtab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nsplat) return;
    using D = Dual<double, K>;
    const double* p = params + 21LL * i;
    D q[21];
    for (int r = 0; r < 21; ++r) {
        q[r] = D(p[r]);
        for (int k = 0; k < K; ++k) q[r].d[k] = dirs[k * dir_stride + 21LL * i + r];
    }
    const double* t0 = tab + (long long)i * ST_COUNT;
    const double* g = gtab + (long long)i * GT_COUNT;
    D o[ST_COUNT];
    for (int e = 0; e < ST_COUNT; ++e) o[e] = D(t0[e]);
    o[ST_CX] = q[0]; o[ST_CY] = q[1]; o[ST_CZ] = q[2];
    o[ST_T0] = q[10]; o[ST_OMEGA] = q[20];
    o[ST_ES1] = exp(-q[3]); o[ST_ES2] = exp(-q[4]); o[ST_ES3] = exp(-q[5]);
    const D n = sqrt(q[6] * q[6] + q[7] * q[7] + q[8] * q[8] + q[9] * q[9]);
    const D w = q[6] / n, x = q[7] / n, y = q[8] / n, z = q[9] / n;
    o[ST_R0] = 1.0 - 2.0 * (y * y + z * z); o[ST_R1] = 2.0 * (x * y - w * z); o[ST_R2] = 2.0 * (x * z + w * y);
    o[ST_R3] = 2.0 * (x * y + w * z); o[ST_R4] = 1.0 - 2.0 * (x * x + z * z); o[ST_R5] = 2.0 * (y * z - w * x);
    o[ST_R6] = 2.0 * (x * z - w * y); o[ST_R7] = 2.0 * (y * z + w * x); o[ST_R8] = 1.0 - 2.0 * (x * x + y * y);
    o[ST_INVW] = exp(-q[11]);
    o[ST_NE] = exp(q[12]);
    o[ST_TE] = exp(q[13]);
    for (int k = 0; k < K; ++k) { o[ST_F0].d[k] = g[GT_DF0] * q[13].d[k]; o[ST_KR].d[k] = g[GT_DKR] * q[13].d[k]; }
    o[ST_BMAG] = exp(q[14]);
    if (t0[ST_BZERO] == 0.0) {
        o[ST_BHX] = sin(q[15]) * cos(q[16]); o[ST_BHY] = sin(q[15]) * sin(q[16]); o[ST_BHZ] = cos(q[15]);
    }
    o[ST_U1] = q[17]; o[ST_U2] = q[18]; o[ST_U3] = q[19];
    Dual<S, K>* out = dtab + (long long)i * ST_COUNT;
    for (int e = 0; e < ST_COUNT; ++e) {
        out[e].v = S(o[e].v);
        for (int k = 0; k < K; ++k) out[e].d[k] = S(o[e].d[k]);
    }
}

// The consumer of the JVP: RadiativeTransport on the dual table (transport.jl:171-198, step.jl:347).
template <class S, int K>
struct JvpSink {
    using D = Dual<S, K>;
    const D* tab; int ntot;
    S t_obs, nu, Lnu, a, rh_lo, dtau, alpha, beta, eta, lam, a_sin_tho, slab;
    int nmax;
    int lnL_dir;      // >= 0: the direction that carries d/d(ln L) (the step length scales with L)
    S reach2 = S(3e38f);   // table_reach2: farther samples weigh no splat
    D P[16], Sv[4];
    S zprev; int wn; bool inside, crossed, zset;

    __device__ void init() {
        for (int q = 0; q < 16; ++q) P[q] = D(S((q % 5 == 0) ? 1 : 0));
        for (int q = 0; q < 4; ++q) Sv[q] = D(S(0));
        wn = 0; inside = false; crossed = false; zset = false; zprev = S(0);
    }
    __device__ void wind(S z) {   // step.jl:379-398
        if (!zset) { zprev = z; zset = true; inside = fabs(z) < slab; crossed = false; return; }
        bool inside_now = fabs(z) < slab;
        bool crossing = zprev * z < S(0);
        if (inside || inside_now) {
            crossed = crossed || crossing;
            if (inside && !inside_now) { if (crossed) wn += 1; crossed = false; }
            else if (!inside && inside_now) { crossed = crossing; }
            inside = inside_now;
        } else if (crossing) {
            wn += 1;
        }
        zprev = z;
    }
    __device__ void operator()(int, const Sample<double>& s64) {
        const S r = S(s64.r), th = S(s64.theta), ph = S(s64.phi), ts = S(s64.t);
        if (!(s64.ok && r > rh_lo)) return;
        if (nmax >= 0) {
            wind(r * cos(th));
            if (wn > nmax) return;
        }
        S x, y, z, sth, cth;
        ks_coords(a, r, th, ph, x, y, z, sth, cth);
        emit(x, y, z, ts, r, sth, cth, s64.nur, s64.nutheta);
    }
    // one sample of the FP32 stream (k_stream: position, lookback time, r, sin/cos theta, flags)
    __device__ void stream_sample(bool usable, S x, S y, S z, S ts, S r, S sth, S cth, bool nur, bool nuth) {
        if (!usable) return;
        if (nmax >= 0) {
            wind(r * cth);
            if (wn > nmax) return;
        }
        emit(x, y, z, ts, r, sth, cth, nur, nuth);
    }
    __device__ void emit(S x, S y, S z, S ts, S r, S sth, S cth, bool nur, bool nuth) {
        if (x * x + y * y + z * z > reach2) return;   // no splat reaches the sample: no element, no step
        const S t = t_obs - ts;
        D in[11];
        for (int q = 0; q < 11; ++q) in[q] = D(S(0));
        bool active = false, have_frame = false;
        SampleFrame<D> F;
        const S rho = sqrt(x * x + y * y);
        for (int i = 0; i < ntot; ++i) {
            const D* p = tab + (long long)i * ST_COUNT;
            // the circle of the pattern rotation, on values first (exact: outside it the support test fails too)
            const S dr = rho - p[ST_RHO].v, dz = z - p[ST_CZ].v;
            if (dr * dr + dz * dz > p[ST_SUPP].v) continue;
            D q;
            if (!splat_exponent(p, D(t), D(x), D(y), D(z), true, q)) continue;
            const D G = exp(-q);
            if (!(G > S(kWEIGHT_CUTOFF))) continue;
            if (!have_frame) {
                const SampleFrame<S> F0 = sample_frame(a, r, S(0), sth, cth, eta, lam, nur, nuth);
                for (int k = 0; k < 4; ++k) { F.pu[k] = D(F0.pu[k]); F.pz[k] = D(F0.pz[k]); }
                F.lapse_inv = D(F0.lapse_inv); F.om_lapse = D(F0.om_lapse); F.sDS = D(F0.sDS); F.misS = D(F0.misS); F.ivarpi = D(F0.ivarpi);
                F.r = D(F0.r); F.sth = D(F0.sth); F.cth = D(F0.cth); F.a = D(F0.a);
                have_frame = true;
            }
            const LFrame<D> lf = local_frame(F, p[ST_U1], p[ST_U2], p[ST_U3], p[ST_BHX], p[ST_BHY], p[ST_BHZ], p[ST_BZERO] != S(0),
                                             D(alpha), D(beta), D(a_sin_tho));
            const D nuf = D(nu) / lf.g;
            D sbv, cbv;
            if constexpr (is_f32<S>) pitch_sc(lf.cosB, sbv, cbv);
            else { const D thb = safe_acos(lf.cosB); sbv = sin(thb); cbv = cos(thb); }
            const Coef<D> cf = thermal_cs(p[ST_NE] * G, p[ST_TE], p[ST_F0], p[ST_KR], p[ST_BMAG], nuf, sbv, cbv);
            if (!(cf.jI > S(0) || cf.aI > S(0) || cf.rQ != S(0) || cf.rV != S(0))) continue;
            const D fe = cap_factor(cf.jI, cf.jQ, cf.jV, D(S(0.99)));
            const D fa = cap_factor(cf.aI, cf.aQ, cf.aV, D(S(0.99)));
            const D nh = nuf / S(kNU0);
            const D i2 = D(S(1)) / (nh * nh);
            const D s2c = lf.s2c, c2c = lf.c2c;
            const D jQ = cf.jQ * fe * i2, aQ = cf.aQ * fa * nh, rQ = cf.rQ * nh;
            in[0] += cf.jI * i2; in[1] += jQ * c2c; in[2] += jQ * s2c; in[3] += cf.jV * fe * i2;
            in[4] += nh * cf.aI; in[5] += aQ * c2c; in[6] += aQ * s2c; in[7] += cf.aV * fa * nh;
            in[8] += rQ * c2c; in[9] += rQ * s2c; in[10] += nh * cf.rV;
            active = true;
        }
        if (!active) return;
        const S Sg = r * r + a * a * cth * cth;
        D Dl(Lnu * Sg * dtau);
        if (lnL_dir >= 0) Dl.d[lnL_dir] = Dl.v;
        D O[16], E[4];
        transfer_step(c_moments, in, in + 4, in + 8, Dl, O, E);
        D Pn[16];
        for (int rr = 0; rr < 4; ++rr) {
            Sv[rr] += P[4 * rr] * E[0] + P[4 * rr + 1] * E[1] + P[4 * rr + 2] * E[2] + P[4 * rr + 3] * E[3];
            for (int q = 0; q < 4; ++q)
                Pn[4 * rr + q] = P[4 * rr] * O[q] + P[4 * rr + 1] * O[4 + q] + P[4 * rr + 2] * O[8 + q] + P[4 * rr + 3] * O[12 + q];
        }
        for (int q = 0; q < 16; ++q) P[q] = Pn[q];
    }
};

// One thread per (ray, combination): the image's K directional derivatives (sorted order)
// out[((d * ncombo + c) * npix + j) * 4 + s], and the image itself in img.
template <class S, int K>
__global__ void __launch_bounds__(64) k_jvp(PlanView P, Spacetime st, long long npix, const Dual<S, K>* __restrict__ dtab, int ntot,
                                            const double* __restrict__ ct, const double* __restrict__ cnu, int ncombo, double L, int nmax,
                                            double slab, double* __restrict__ img, double* __restrict__ out, int lnL_dir) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= npix * ncombo) return;
    const long long j = idx % npix;
    const int c = int(idx / npix);
    MarchRay<double> R = load_ray<double>(P, st, j);
    JvpSink<S, K> sink;
    sink.tab = dtab; sink.ntot = ntot;
    sink.t_obs = S(ct[c]); sink.nu = S(cnu[c]);
    const double nh = cnu[c] / kNU0;
    sink.Lnu = S(L / nh);
    sink.a = S(st.a); sink.rh_lo = S(st.rh * (1 + 1e-3)); sink.dtau = S(R.dtau);
    sink.alpha = S(P.get(PF_ALPHA, j)); sink.beta = S(P.get(PF_BETA, j)); sink.eta = S(R.eta); sink.lam = S(R.lam);
    sink.a_sin_tho = S(st.a * sin(st.thetao)); sink.slab = S(slab); sink.nmax = nmax;
    sink.lnL_dir = lnL_dir;
    sink.init();
    double rt, rp;
    march(P, st, j, R, sink, rt, rp);
    const double n3 = nh * nh * nh;
    for (int s = 0; s < 4; ++s) {
        img[(c * npix + j) * 4 + s] = double(sink.Sv[s].v) * n3;
        for (int d = 0; d < K; ++d) out[(((long long)d * ncombo + c) * npix + j) * 4 + s] = double(sink.Sv[s].d[d]) * n3;
    }
}

// The mixed J v over the FP32 sample stream of k_stream: one thread per (segment of the samples, combination, ray),
// which composes the segment's (P, S) on duals; k_jvp_combine joins the segments. Bound by the dual pair evaluations
// of the rays that cross splats: one thread per whole ray ran 71 ms for two directions on 96 x 96 rays x 256 samples,
// two warps per SM deep. The first sample past the half-orbit cutoff is `kstop` (null: none).
template <int K>
__global__ void __launch_bounds__(64, 8) k_jvp_stream(PlanView P, Spacetime st, long long npix, const Dual<float, K>* __restrict__ dtab, int ntot,
                                                   const double* __restrict__ ct, const double* __restrict__ cnu, int ncombo, double L,
                                                   const int* __restrict__ kstop, int nseg, int seg_len, const float* __restrict__ stream,
                                                   float* __restrict__ part, int lnL_dir) {
    __shared__ float s_reach;
    const float reach2 = table_reach2(dtab, ntot, &s_reach);   // before any thread leaves: it has block barriers
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= npix * ncombo * nseg) return;
    const long long j = idx % npix;
    const int c = int(idx / npix % ncombo), seg = int(idx / npix / ncombo);
    const long long npad = P.npad;
    JvpSink<float, K> sink;
    sink.tab = dtab; sink.ntot = ntot; sink.reach2 = reach2;
    sink.t_obs = float(ct[c]); sink.nu = float(cnu[c]);
    const double nh = cnu[c] / kNU0;
    sink.Lnu = float(L / nh);
    sink.a = float(st.a); sink.rh_lo = float(st.rh * (1 + 1e-3)); sink.dtau = float(P.get(PF_DTAU, j));
    sink.alpha = float(P.get(PF_ALPHA, j)); sink.beta = float(P.get(PF_BETA, j));
    sink.eta = float(P.get(PF_ETA, j)); sink.lam = float(P.get(PF_LAM, j));
    sink.a_sin_tho = float(st.a * sin(st.thetao)); sink.slab = 0.f; sink.nmax = -1;
    sink.lnL_dir = lnL_dir;
    sink.init();
    int k1 = min(int(P.get(PF_NSAMP, j)) + 1, 1 + (seg + 1) * seg_len);
    if (kstop) k1 = min(k1, kstop[j]);
    const float* sp = stream + (long long)seg * seg_len * SM_COUNT * npad + j;
    for (int k = 1 + seg * seg_len; k < k1; ++k, sp += SM_COUNT * npad) {
        const unsigned flags = __float_as_uint(sp[SM_FLAGS * npad]);
        sink.stream_sample((flags & 8u) != 0u, sp[SM_X * npad], sp[SM_Y * npad], sp[SM_Z * npad], sp[SM_T * npad], sp[SM_R * npad],
                           sp[SM_STH * npad], sp[SM_CTH * npad], (flags & 2u) != 0u, (flags & 4u) != 0u);
    }
    // [seg][combination][20 (K + 1)][ray]
    float* o = part + (idx / npix) * (20 * (K + 1)) * npix + j;
    for (int q = 0; q < 20; ++q) {
        const Dual<float, K>& x = q < 16 ? sink.P[q] : sink.Sv[q - 16];
        o[(long long)q * (K + 1) * npix] = x.v;
        for (int d = 0; d < K; ++d) o[(long long)(q * (K + 1) + 1 + d) * npix] = x.d[d];
    }
}

// The segments of a ray front to back (S = S_0 + P_0 (S_1 + ...)) on duals, and the observed Stokes vector (x nuhat^3).
template <int K>
__global__ void k_jvp_combine(long long npix, int ncombo, int nseg, const double* __restrict__ cnu, const float* __restrict__ part,
                              double* __restrict__ img, double* __restrict__ out) {
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= npix * ncombo) return;
    const long long j = idx % npix, c = idx / npix;
    double S[4][K + 1];
    for (int r = 0; r < 4; ++r)
        for (int d = 0; d <= K; ++d) S[r][d] = 0.0;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const float* p = part + ((long long)sg * ncombo + c) * (20 * (K + 1)) * npix + j;
        double T[4][K + 1];
        for (int r = 0; r < 4; ++r) {
            for (int d = 0; d <= K; ++d) T[r][d] = p[(long long)((16 + r) * (K + 1) + d) * npix];
            for (int q = 0; q < 4; ++q) {
                const double pv = p[(long long)((4 * r + q) * (K + 1)) * npix];
                T[r][0] += pv * S[q][0];
                for (int d = 1; d <= K; ++d) T[r][d] += pv * S[q][d] + double(p[(long long)((4 * r + q) * (K + 1) + d) * npix]) * S[q][0];
            }
        }
        for (int r = 0; r < 4; ++r)
            for (int d = 0; d <= K; ++d) S[r][d] = T[r][d];
    }
    const double nh = cnu[c] / kNU0, n3 = nh * nh * nh;
    for (int r = 0; r < 4; ++r) {
        img[(c * npix + j) * 4 + r] = S[r][0] * n3;
        for (int d = 0; d < K; ++d) out[(((long long)d * ncombo + c) * npix + j) * 4 + r] = S[r][1 + d] * n3;
    }
}

}  // namespace

namespace {

// A = J^T J (normal_matrix, gauss_newton.jl:486-494) of a row-major m x n FP64 Jacobian, FP64 tiles
// of 32 x 32 with the shared k-slab; only the upper triangle's tiles are computed and mirrored.
__global__ void k_normal_fp64(long long m, int n, const double* __restrict__ J, double* __restrict__ A) {
    __shared__ double Ja[32][33], Jb[32][33];
    const int bi = blockIdx.y, bj = blockIdx.x;
    if (bj < bi) return;
    const int tx = threadIdx.x, ty = threadIdx.y;   // 32 x 8
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long k0 = 0; k0 < m; k0 += 32) {
        for (int q = 0; q < 4; ++q) {
            const int kk = ty + 8 * q;
            const long long r = k0 + kk;
            const int ca = bi * 32 + tx, cb = bj * 32 + tx;
            Ja[kk][tx] = (r < m && ca < n) ? J[r * n + ca] : 0.0;
            Jb[kk][tx] = (r < m && cb < n) ? J[r * n + cb] : 0.0;
        }
        __syncthreads();
        for (int kk = 0; kk < 32; ++kk) {
            const double b = Jb[kk][tx];
            for (int q = 0; q < 4; ++q) acc[q] += Ja[kk][ty + 8 * q] * b;
        }
        __syncthreads();
    }
    for (int q = 0; q < 4; ++q) {
        const int i = bi * 32 + ty + 8 * q, j = bj * 32 + tx;
        if (i < n && j < n) { A[(long long)i * n + j] = acc[q]; A[(long long)j * n + i] = acc[q]; }
    }
}

// row-major m x n (double) -> the split GEMM operand y[n][ld] (row c holds column c of x)
__global__ void k_transpose_split(long long m, int n, const double* __restrict__ x, float* __restrict__ hi, float* __restrict__ lo,
                                  long long ld) {
    __shared__ float t[32][33];
    const long long r0 = (long long)blockIdx.y * 32;
    const int c0 = blockIdx.x * 32;
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const long long r = r0 + q;
        const int cc = c0 + threadIdx.x;
        t[q][threadIdx.x] = (r < m && cc < n) ? float(x[r * n + cc]) : 0.f;
    }
    __syncthreads();
    for (int q = threadIdx.y; q < 32; q += blockDim.y) {
        const int cc = c0 + q;
        const long long r = r0 + threadIdx.x;
        if (cc < n && r < m) ksdft::split_store(hi, lo, (long long)cc * ld + r, t[threadIdx.x][q]);
    }
}
__global__ void k_to_f64(long long n, const float* __restrict__ x, double* __restrict__ y) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q < n) y[q] = double(x[q]);
}

}  // namespace
