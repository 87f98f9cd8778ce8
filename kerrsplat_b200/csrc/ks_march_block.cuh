// ks_march_block.cuh -- the march of 32 rays by a block of four warps, eight samples at a time: the same samples as
// march_impl (ks_march.cuh), operation for operation, with what does not have to be serial taken out of the chain.
//
// A sample of march_impl is one chain of four addition-theorem steps, two evaluations of the rates, three logarithms,
// two arctangents and the caller's work: some 3.4 us (FP32 march) to 8 us (FP64, thin image) a sample for a thread
// alone, which is all a small screen has. Only the Jacobi states and the running sums of t~ and phi depend on the
// sample before. Here, for each run of eight samples (lane = ray):
//   1. warp 0 steps the radial states and warp 1 the polar ones into shared memory;
//   2. every warp evaluates two samples' points (end and middle), then their interval increments;
//   3. warp 0 adds the increments up, anchor by anchor;
//   4. every warp hands two samples to the caller.
// Each phase also holds only its own part of the ray's constants in registers (they come from shared memory).
#pragma once
#include "ks_march.cuh"

namespace ks {

constexpr int kMarchRun = 8, kMarchWarps = 4;

// What the phases keep in shared memory.
template <class T>
struct MarchShared {
    using PT = GeoT<T>;
    // ray constants: in the geometry's precision, in the march's
    enum { G_K, G_M0, G_M1, G_M2, G_M3, G_PMU, G_PSCALE, G_SQRTUP, G_UM, G_UPMUM, G_PSIGN, G_VABSALPHA, G_VALPHA2, G_VABSBETA, G_DRSN, G_DRCN, G_DRDN,
           G_DTSN, G_DTCN, G_DTDN, G_COUNT };
    enum { D_TAUVALID, D_DTAU, D_FO, D_COUNT };
    enum { C_TEMPFAC, C_POFFSET, C_LAM, C_ETA, C_SP, C_SM, C_QT, C_QTM, C_QPHI, C_QPHIM, C_R4, C_QC, C_QN, C_SQRTEPS, C_GC, C_MP, C_K2, C_COUNT };
    double d[D_COUNT][32];
    PT g[G_COUNT][32];
    PT state[kMarchRun][4][3][32];           // radial middle, radial end, polar middle, polar end
    PT sum[kMarchRun][2][32];                // increments, then t~ and phi
    T c[C_COUNT][32];
    T point[kMarchRun + 1][4][32];           // r, the rates of t and phi, polar_closed; slot 0: the sample before the run
    T cth[kMarchRun][32];
    unsigned char bits[kMarchRun][32];       // 1 ok, 2 inbound, 4 toward the pole
    unsigned char rcase[32];                 // root case, 8 vortical, 16 scattering
    int turn_k[32];
};

template <class T>
__device__ __forceinline__ MarchRay<T> shared_ray(const MarchShared<T>& s, const Spacetime& st, int lane) {
    using M = MarchShared<T>;
    using PT = GeoT<T>;
    MarchRay<T> R;
    R.rcase = s.rcase[lane] & 7; R.vortical = (s.rcase[lane] & 8) != 0; R.scattering = (s.rcase[lane] & 16) != 0;
    R.tau_valid = s.d[M::D_TAUVALID][lane]; R.dtau = s.d[M::D_DTAU][lane]; R.fo_d = s.d[M::D_FO][lane];
    R.k = s.g[M::G_K][lane]; R.m0 = s.g[M::G_M0][lane]; R.m1 = s.g[M::G_M1][lane]; R.m2 = s.g[M::G_M2][lane]; R.m3 = s.g[M::G_M3][lane];
    R.pmu = s.g[M::G_PMU][lane]; R.pscale = s.g[M::G_PSCALE][lane]; R.sqrt_up = s.g[M::G_SQRTUP][lane]; R.um = s.g[M::G_UM][lane];
    R.up_m_um = s.g[M::G_UPMUM][lane]; R.psign = s.g[M::G_PSIGN][lane];
    R.vabsalpha = s.g[M::G_VABSALPHA][lane]; R.valpha2 = s.g[M::G_VALPHA2][lane]; R.vabsbeta = s.g[M::G_VABSBETA][lane];
    R.dr = {s.g[M::G_DRSN][lane], s.g[M::G_DRCN][lane], s.g[M::G_DRDN][lane]};
    R.dth = {s.g[M::G_DTSN][lane], s.g[M::G_DTCN][lane], s.g[M::G_DTDN][lane]};
    R.tempfac = s.c[M::C_TEMPFAC][lane]; R.poffset = s.c[M::C_POFFSET][lane]; R.lam = s.c[M::C_LAM][lane]; R.eta = s.c[M::C_ETA][lane];
    R.sp = s.c[M::C_SP][lane]; R.sm = s.c[M::C_SM][lane]; R.Qt = s.c[M::C_QT][lane]; R.Qtm = s.c[M::C_QTM][lane];
    R.Qphi = s.c[M::C_QPHI][lane]; R.Qphim = s.c[M::C_QPHIM][lane]; R.r4 = s.c[M::C_R4][lane]; R.qC = s.c[M::C_QC][lane]; R.qn = s.c[M::C_QN][lane];
    R.sqrt_eps = s.c[M::C_SQRTEPS][lane]; R.gc = s.c[M::C_GC][lane]; R.mp = s.c[M::C_MP][lane]; R.K2 = s.c[M::C_K2][lane];
    R.a = T(st.a); R.rp = T(st.rp); R.rmn = T(st.rmn); R.vabscos = PT(st.abscos); R.vcos2 = PT(st.cos2); R.pa = PT(st.a);
    R.turn_k = s.turn_k[lane];
    return R;
}

// March samples [k_begin, k_end) of the block's rays (lane = ray j; `live` false past the last ray) and call
// f(k, sample) for each, a thread every fourth sample. All 128 threads call it; `s` is the block's. With RESID the
// largest |quadrature - anchor| of the range's intervals comes back in warp 0 (march_impl's rule at the range's end).
template <bool RESID, class T, class F>
__device__ __forceinline__ void march_block(const PlanView& P, const Spacetime& st, long long j, bool live, int k_begin, int k_end, MarchShared<T>& s,
                                            F& f, double& resid_t, double& resid_phi) {
    using M = MarchShared<T>;
    using PT = GeoT<T>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int Man, nanch, nsamp;
    long long aoff;
    double dtau;
    {
        const MarchRay<T> R = load_ray<T>(P, st, j);
        Man = R.Manchor; nanch = R.nanch; nsamp = live ? R.nsamp : 0; aoff = R.anchor_off; dtau = R.dtau;
        if (warp == 0) {
            s.rcase[lane] = (unsigned char)(R.rcase | (R.vortical ? 8 : 0) | (R.scattering ? 16 : 0));
            s.turn_k[lane] = R.turn_k;
            s.d[M::D_TAUVALID][lane] = R.tau_valid; s.d[M::D_DTAU][lane] = R.dtau; s.d[M::D_FO][lane] = R.fo_d;
        } else if (warp == 1) {
            s.g[M::G_K][lane] = R.k; s.g[M::G_M0][lane] = R.m0; s.g[M::G_M1][lane] = R.m1; s.g[M::G_M2][lane] = R.m2; s.g[M::G_M3][lane] = R.m3;
            s.g[M::G_PMU][lane] = R.pmu; s.g[M::G_PSCALE][lane] = R.pscale; s.g[M::G_SQRTUP][lane] = R.sqrt_up; s.g[M::G_UM][lane] = R.um;
            s.g[M::G_UPMUM][lane] = R.up_m_um; s.g[M::G_PSIGN][lane] = R.psign;
        } else if (warp == 2) {
            s.g[M::G_VABSALPHA][lane] = R.vabsalpha; s.g[M::G_VALPHA2][lane] = R.valpha2; s.g[M::G_VABSBETA][lane] = R.vabsbeta;
            s.g[M::G_DRSN][lane] = R.dr.sn; s.g[M::G_DRCN][lane] = R.dr.cn; s.g[M::G_DRDN][lane] = R.dr.dn;
            s.g[M::G_DTSN][lane] = R.dth.sn; s.g[M::G_DTCN][lane] = R.dth.cn; s.g[M::G_DTDN][lane] = R.dth.dn;
        } else {
            s.c[M::C_TEMPFAC][lane] = R.tempfac; s.c[M::C_POFFSET][lane] = R.poffset; s.c[M::C_LAM][lane] = R.lam; s.c[M::C_ETA][lane] = R.eta;
            s.c[M::C_SP][lane] = R.sp; s.c[M::C_SM][lane] = R.sm; s.c[M::C_QT][lane] = R.Qt; s.c[M::C_QTM][lane] = R.Qtm;
            s.c[M::C_QPHI][lane] = R.Qphi; s.c[M::C_QPHIM][lane] = R.Qphim; s.c[M::C_R4][lane] = R.r4; s.c[M::C_QC][lane] = R.qC; s.c[M::C_QN][lane] = R.qn;
            s.c[M::C_SQRTEPS][lane] = R.sqrt_eps; s.c[M::C_GC][lane] = R.gc; s.c[M::C_MP][lane] = R.mp; s.c[M::C_K2][lane] = R.K2;
        }
    }
    if (k_end > nsamp + 1) k_end = nsamp + 1;
    const bool any = k_begin < k_end;
    int k_stop = k_end + ((RESID && k_end <= nsamp && (k_end - 1) % Man == 0) ? 1 : 0);
    int m0 = (k_begin - 1) / Man;
    if (m0 > nanch - 1) m0 = nanch - 1;
    int ka = 1 + m0 * Man;   // the anchor the ray starts from
    if (!any) { ka = 1 << 30; k_stop = 0; }
    const int kfirst = __reduce_min_sync(0xffffffffu, ka), klast = __reduce_max_sync(0xffffffffu, k_stop);
    const double* A = P.anchors + aoff * AF_COUNT;
    JS<PT> x{PT(0), PT(1), PT(1)};           // warp 0: radial, warp 1: polar
    int m = m0;                              // warps 0, 1: the last anchor taken by the states
    int ms = m0;                             // warp 0: ... by the sums
    PT t = PT(0), phi = PT(0);
    double rt = 0.0, rphi = 0.0;
    __syncthreads();
    for (int kb = kfirst; kb < klast; kb += kMarchRun) {
        // 1. the states
        if (warp < 2) {
            const JS<PT> step = warp == 0 ? JS<PT>{s.g[M::G_DRSN][lane], s.g[M::G_DRCN][lane], s.g[M::G_DRDN][lane]}
                                          : JS<PT>{s.g[M::G_DTSN][lane], s.g[M::G_DTCN][lane], s.g[M::G_DTDN][lane]};
            const PT mu = warp == 0 ? s.g[M::G_K][lane] : s.g[M::G_PMU][lane];
            const int off = warp == 0 ? AF_XR_SN : AF_XT_SN;
#pragma unroll 1
            for (int c = 0; c < kMarchRun; ++c) {
                const int k = kb + c;
                if (k < ka || k >= k_stop) continue;
                if (k == ka) {
                    x = load_js<PT>(A + (long long)m * AF_COUNT, off);
                } else {
                    x = jstep(x, step, mu);
                    s.state[c][2 * warp][0][lane] = x.sn; s.state[c][2 * warp][1][lane] = x.cn; s.state[c][2 * warp][2][lane] = x.dn;
                    if (k == 1 + (m + 1) * Man) {
                        ++m;
                        x = load_js<PT>(A + (long long)m * AF_COUNT, off);
                    } else {
                        x = jstep(x, step, mu);
                    }
                }
                s.state[c][2 * warp + 1][0][lane] = x.sn; s.state[c][2 * warp + 1][1][lane] = x.cn; s.state[c][2 * warp + 1][2][lane] = x.dn;
            }
        }
        __syncthreads();
        // 2. the points, then the increments of this thread's samples
        const double h = dtau / 2.0;
        T mgt[kMarchRun / kMarchWarps], mgp[kMarchRun / kMarchWarps];
        {
            const MarchRay<T> R = shared_ray(s, st, lane);
#pragma unroll
            for (int q = 0; q < kMarchRun / kMarchWarps; ++q) {
                const int c = q * kMarchWarps + warp, k = kb + c;
                mgt[q] = mgp[q] = T(0);
                if (k < ka || k >= k_stop) continue;
                const JS<PT> xr{s.state[c][1][0][lane], s.state[c][1][1][lane], s.state[c][1][2][lane]};
                const JS<PT> xt{s.state[c][3][0][lane], s.state[c][3][1][lane], s.state[c][3][2][lane]};
                const double tb = k * dtau;
                const Point<T> p = ray_point(R, xr, xt, tb);
                s.point[c + 1][0][lane] = p.r; s.point[c + 1][1][lane] = p.gt; s.point[c + 1][2][lane] = p.gphi;
                s.point[c + 1][3][lane] = polar_closed(R, tb, p.sn, p.cn);
                s.cth[c][lane] = p.cth;
                s.bits[c][lane] = (unsigned char)((((tb <= R.tau_valid) && visible(R, p.cthp)) ? 1 : 0) | (p.nur ? 2 : 0) | (p.nuth ? 4 : 0));
                if (k > ka) {
                    const JS<PT> yr{s.state[c][0][0][lane], s.state[c][0][1][lane], s.state[c][0][2][lane]};
                    const JS<PT> yt{s.state[c][2][0][lane], s.state[c][2][1][lane], s.state[c][2][2][lane]};
                    const Point<T> pm = ray_point(R, yr, yt, (k - 1) * dtau + h);
                    mgt[q] = pm.gt; mgp[q] = pm.gphi;
                }
            }
        }
        __syncthreads();
        {
            const MarchRay<T> R = shared_ray(s, st, lane);
#pragma unroll
            for (int q = 0; q < kMarchRun / kMarchWarps; ++q) {
                const int c = q * kMarchWarps + warp, k = kb + c;
                if (k <= ka || k >= k_stop) continue;
                const double ta = (k - 1) * dtau, tb = k * dtau;
                Point<T> pa, pm, pb;
                pa.r = s.point[c][0][lane]; pa.gt = s.point[c][1][lane]; pa.gphi = s.point[c][2][lane];
                pb.r = s.point[c + 1][0][lane]; pb.gt = s.point[c + 1][1][lane]; pb.gphi = s.point[c + 1][2][lane];
                pm.gt = mgt[q]; pm.gphi = mgp[q];
                const T pca = s.point[c][3][lane], pcb = s.point[c + 1][3][lane];
                PT it, ip;
                if (k == R.turn_k) {
                    const double* pf = P.f;
                    const long long np = P.npad;
                    const JS<PT> p1r = {PT(pf[PF_P1R_SN * np + j]), PT(pf[PF_P1R_CN * np + j]), PT(pf[PF_P1R_DN * np + j])};
                    const JS<PT> p1t = {PT(pf[PF_P1T_SN * np + j]), PT(pf[PF_P1T_CN * np + j]), PT(pf[PF_P1T_DN * np + j])};
                    const JS<PT> p2r = {PT(pf[PF_P2R_SN * np + j]), PT(pf[PF_P2R_CN * np + j]), PT(pf[PF_P2R_DN * np + j])};
                    const JS<PT> p2t = {PT(pf[PF_P2T_SN * np + j]), PT(pf[PF_P2T_CN * np + j]), PT(pf[PF_P2T_DN * np + j])};
                    const JS<PT> ptt = {PT(pf[PF_PTT_SN * np + j]), PT(pf[PF_PTT_CN * np + j]), PT(pf[PF_PTT_DN * np + j])};
                    const double fo = R.fo_d;
                    const Point<T> pt = turning_point(R, ptt);
                    const Point<T> p1 = ray_point(R, p1r, p1t, (ta + fo) / 2.0), p2 = ray_point(R, p2r, p2t, (fo + tb) / 2.0);
                    const T pct = polar_closed(R, fo, pt.sn, pt.cn);
                    T It1, Ip1, It2, Ip2;
                    increment(R, pa, p1, pt, ta, fo, pca, pct, It1, Ip1);
                    increment(R, pt, p2, pb, fo, tb, pct, pcb, It2, Ip2);
                    it = PT(It1) + PT(It2); ip = PT(Ip1) + PT(Ip2);
                } else {
                    T It, Ip;
                    increment(R, pa, pm, pb, ta, tb, pca, pcb, It, Ip);
                    it = PT(It); ip = PT(Ip);
                }
                s.sum[c][0][lane] = it; s.sum[c][1][lane] = ip;
            }
        }
        __syncthreads();
        // 3. the running sums, reset to the anchors; the run's last point in front of the next run
        if (warp == 0) {
#pragma unroll 1
            for (int c = 0; c < kMarchRun; ++c) {
                const int k = kb + c;
                if (k < ka || k >= k_stop) continue;
                if (k == ka) {
                    const double* Am = A + (long long)ms * AF_COUNT;
                    t = PT(Am[AF_T]); phi = PT(Am[AF_PHI]);
                } else {
                    t += s.sum[c][0][lane]; phi += s.sum[c][1][lane];
                    if (k == 1 + (ms + 1) * Man) {
                        ++ms;
                        const double* Am = A + (long long)ms * AF_COUNT;
                        if (Am[AF_OK] != 0.0) {
                            const double at = Am[AF_T], ap = Am[AF_PHI];
                            if constexpr (RESID) {
                                rt = fmax(rt, fabs(double(t) - at));
                                rphi = fmax(rphi, fabs(double(phi) - ap));
                            }
                            t = PT(at); phi = PT(ap);
                        }
                    }
                }
                s.sum[c][0][lane] = t; s.sum[c][1][lane] = phi;
            }
        } else if (warp == 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) s.point[0][q][lane] = s.point[kMarchRun][q][lane];
        }
        __syncthreads();
        // 4. the samples
#pragma unroll 1
        for (int c = warp; c < kMarchRun; c += kMarchWarps) {
            const int k = kb + c;
            if (k < ka || k < k_begin || k >= k_end) continue;
            const unsigned b = s.bits[c][lane];
            Sample<T> o;
            o.t = T(s.sum[c][0][lane]); o.r = s.point[c + 1][0][lane]; o.theta = T(0); o.cos_theta = s.cth[c][lane]; o.phi = T(s.sum[c][1][lane]);
            o.nur = (b & 2u) != 0; o.nutheta = (b & 4u) != 0; o.ok = (b & 1u) != 0;
            f(k, o);
        }
    }
    resid_t = rt;
    resid_phi = rphi;
}

}  // namespace ks
