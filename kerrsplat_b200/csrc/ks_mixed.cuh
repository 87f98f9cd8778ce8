// ks_mixed.cuh -- the sample stream and what its consumers share: the bounds of a work unit and its candidate
// splats, the bulk staging of the splat tables, the block scan.
//
// k_stream marches every ray once (the recurrence and the quadrature, re-anchored to the FP64 table every M
// samples) into a sample stream that every frame, frequency and parameter set reads.
#pragma once
#include "ks_march_block.cuh"
#include "ks_transfer.cuh"

namespace ks {

constexpr double kQCUT = 13.815510557964274;   // -ln(WEIGHT_CUTOFF): G > 1e-6 <=> q < QCUT

constexpr int kMaxSplatWords = 16;              // the FP32 transport takes up to 512 splats

// The bounds of a work unit's samples (quasi-Cartesian KS box, cylindrical radius and height, and the
// range of their lookback times) and the splats whose support can reach them: a
// pattern-rotating splat's support lies within its support radius of the circle its centre runs on
// (rho = ST_RHO, z = ST_CZ), and within it of the arc its centre covers over the unit's emission times
// (the centre's angle is phi_0 + omega (t - t0)); a knot splat's within its bounding sphere (centre
// ST_CX..CZ, radius^2 ST_RHO). Splats outside are below the weight cutoff at every sample of the unit,
// so the per-sample tests skip them (the same result, fewer tests).
struct UnitBox { float xlo, xhi, ylo, yhi, zlo, zhi, rlo, rhi, slo, shi; };

// Widen the unit box with one sample (position, cylindrical radius, lookback time).
__device__ __forceinline__ void unit_box_add(UnitBox& b, float x, float y, float z, float s) {
    const float rho = sqrtf(x * x + y * y);
    b.xlo = fminf(b.xlo, x); b.xhi = fmaxf(b.xhi, x); b.ylo = fminf(b.ylo, y); b.yhi = fmaxf(b.yhi, y);
    b.zlo = fminf(b.zlo, z); b.zhi = fmaxf(b.zhi, z); b.rlo = fminf(b.rlo, rho); b.rhi = fmaxf(b.rhi, rho);
    b.slo = fminf(b.slo, s); b.shi = fmaxf(b.shi, s);
}
__device__ __forceinline__ UnitBox unit_box_empty() { return {3e38f, -3e38f, 3e38f, -3e38f, 3e38f, -3e38f, 3e38f, -3e38f, 3e38f, -3e38f}; }

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, d));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    return v;
}

// The squared radius (about the origin of the quasi-Cartesian frame) beyond which no splat of the
// table can weigh a sample: the pattern rotation keeps a centre's distance from the origin, so a
// pattern-rotating splat reaches |c| + sqrt(support); a knot splat reaches its bounding sphere. Padded
// by 1e-3 relative for the FP32 rounding of the positions. Every thread of the block calls it (the
// table in shared or global memory, values or duals); `slot` is a block-shared float.
template <class TAB>
__device__ __forceinline__ float table_reach2(const TAB* tab, int ntot, float* slot) {
    if (threadIdx.x == 0) *slot = 0.f;
    __syncthreads();
    float m = 0.f;
    for (int i = threadIdx.x; i < ntot; i += blockDim.x) {
        const TAB* p = tab + (long long)i * ST_COUNT;
        const float cx = float(value_of(p[ST_CX])), cy = float(value_of(p[ST_CY])), cz = float(value_of(p[ST_CZ]));
        const bool knot = int(value_of(p[ST_KIND])) == KS_KNOT21;
        const float c = sqrtf(cx * cx + cy * cy + cz * cz);
        m = fmaxf(m, c + sqrtf(float(value_of(knot ? p[ST_RHO] : p[ST_SUPP]))));
    }
    atomicMax(reinterpret_cast<int*>(slot), __float_as_int(m));   // non-negative floats order as ints
    __syncthreads();
    const float r = *slot * 1.001f + 1e-3f;
    return r * r;
}

// The warp's union of its lanes' boxes.
__device__ __forceinline__ void unit_box_reduce(UnitBox& b) {
    b.xlo = warp_min(b.xlo); b.xhi = warp_max(b.xhi); b.ylo = warp_min(b.ylo); b.yhi = warp_max(b.yhi);
    b.zlo = warp_min(b.zlo); b.zhi = warp_max(b.zhi); b.rlo = warp_min(b.rlo); b.rhi = warp_max(b.rhi);
    b.slo = warp_min(b.slo); b.shi = warp_max(b.shi);
}

// ---- TMA bulk staging ----------------------------------------------------------------------------

constexpr int kStageWaitLimit = 1 << 22;   // mbarrier polls before a staging copy is declared lost

__device__ __forceinline__ unsigned smem_u32(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }

// Stage `bytes` (a multiple of 16; both addresses 16-byte aligned) from global memory into this CTA's
// shared memory with one TMA bulk copy (cp.async.bulk, no multicast) completing on the mbarrier `bar`.
// Every thread of the block calls it; thread 0 initialises the barrier and issues the copy, all
// threads wait for the barrier's phase 0 with a bounded number of polls. Returns false (the same in
// every thread) when the copy did not land within the limit: the caller records an error and returns.
// With issue == false (a test of the error path) the barrier is armed but no copy is issued, so every
// thread's wait runs out after `limit` polls and the function returns false.
__device__ __forceinline__ bool stage_bulk(void* dst, const void* src, unsigned bytes, unsigned long long* bar, bool issue = true,
                                           int limit = kStageWaitLimit) {
    const unsigned b = smem_u32(bar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(b) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the barrier, visible to the copy engine
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared.b64 st, [%0], %1;\n\t}" ::"r"(b), "r"(bytes) : "memory");
        if (issue)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(b) : "memory");
    }
    unsigned done = 0;
    for (int it = 0; it < limit && !done; ++it)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(b) : "memory");
    return __syncthreads_and(done != 0) != 0;
}

// The sample stream: every sample of every ray, marched once per render (the recurrence and the quadrature
// re-anchored to the FP64 table) and shared by every frame, frequency and parameter set. FP32 values for the
// mixed transport, FP64 for the plain one. Layout [k][field][npad] (k = sample - 1): the lanes of a warp (consecutive sorted rays) read and
// write consecutive addresses.
enum StreamField { SM_X, SM_Y, SM_Z, SM_T, SM_R, SM_STH, SM_CTH, SM_FLAGS, SM_COUNT };

// a sample's flags (1 visible, 2 inbound, 4 toward the pole, 8 usable), kept as the bits of its last field
__device__ __forceinline__ unsigned stream_flags(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned stream_flags(double v) { return unsigned(__double_as_longlong(v)); }
__device__ __forceinline__ void set_stream_flags(float* o, unsigned f) { *o = __uint_as_float(f); }
__device__ __forceinline__ void set_stream_flags(double* o, unsigned f) { *o = __longlong_as_double((long long)f); }

// T: the precision of the march (float: the mixed path; double: FP64 geodesics with the transport in
// FP32, the reference's `precision(cache, Float32)` arrangement, cache.jl:212-232). S: the stream's values.
template <class T, class S>
struct StreamSink {
    S* out;
    long long npad, j;
    T a, rh_lo;
    T rp, rm;       // the horizons
    float afac;     // a / (2 sqrt(1 - a^2))
    // The quasi-Cartesian Kerr-Schild position of ks_coords in the precision of the stream: the sample
    // is FP64 (T = double) but x, y, z are stored in FP32, so the angles go to FP32 trigonometry once
    // phi_KS is reduced into [-pi, pi] in T; sin theta comes from cos theta (sqrt((1 - c)(1 + c)),
    // as accurate as sin(acos c)); r - r_+ and r - r_- are formed in T before the FP32 logarithm.
    __device__ void operator()(int k, const Sample<T>& s) {
        S* o = out + (long long)(k - 1) * SM_COUNT * npad + j;
        const bool usable = s.ok && s.r > rh_lo;
        unsigned flags = (s.ok ? 1u : 0u) | (s.nur ? 2u : 0u) | (s.nutheta ? 4u : 0u) | (usable ? 8u : 0u);
        S x = S(0), y = S(0), z = S(0), sth = S(0), cth = S(0);
        if constexpr (sizeof(S) == 8) {
            // FP64 throughout, sin theta from cos theta (no angle formed)
            if (usable) {
                cth = s.cos_theta;
                sth = sqrt(fmax((1.0 - cth) * (1.0 + cth), 0.0));
                ks_position(a, s.r, sth, cth, s.phi, x, y, z);
            }
        } else if (usable) {
            const T c = s.cos_theta;
            const T st2 = (T(1) - c) * (T(1) + c);
            cth = float(c);
            sth = float(sqrt(st2 > T(0) ? st2 : T(0)));
            const float lg = logf(fabsf(float(s.r - rp + keps<T>()) / float(s.r - rm + keps<T>())));
            const T phks = s.phi + T(afac * lg - atan2f(float(a), float(s.r)));
            const T turns = rint(phks * T(0.15915494309189535));   // 1 / (2 pi)
            const float phr = float(phks - turns * T(6.283185307179586));
            float sp, cp;
            sincosf(phr, &sp, &cp);
            const float r = float(s.r);
            x = r * sth * cp; y = r * sth * sp; z = r * cth;
        }
        o[SM_X * npad] = x; o[SM_Y * npad] = y; o[SM_Z * npad] = z; o[SM_T * npad] = S(s.t);
        o[SM_R * npad] = S(s.r); o[SM_STH * npad] = sth; o[SM_CTH * npad] = cth;
        set_stream_flags(o + SM_FLAGS * npad, flags);
    }
};

// One thread per (ray, segment of seg_len samples starting at an anchor multiple) of the rays [j0, j0 + npix).
// At most 128 registers (four blocks per SM): the FP64 march held 252 and ran 8 warps per SM; capped, 16
// warps per SM hide more of the FP64 latency (4% of the configuration-2 render, same stream). The FP64 stream
// also leaves the anchor residuals of its rays (the largest over the segments).
template <class T, class S>
__global__ void __launch_bounds__(128, 4) k_stream(PlanView P, Spacetime st, long long j0, long long npix, long long npad, int seg_len, int nseg,
                                                   S* __restrict__ out, unsigned long long* __restrict__ resid_t,
                                                   unsigned long long* __restrict__ resid_phi) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= npix * nseg) return;
    const long long j = q % npix;
    const int seg = int(q / npix);
    const int k0 = 1 + seg * seg_len, k1 = min(st.N + 1, k0 + seg_len);
    MarchRay<T> R = load_ray<T>(P, st, j0 + j);
    const double temp = sqrt(1.0 - st.a * st.a);
    StreamSink<T, S> sink{out, npad, j, T(st.a), T(st.rh * (1 + 1e-3)), T(1.0 + temp), T(1.0 - temp), float(st.a / (2.0 * temp))};
    if constexpr (sizeof(S) == 8) {
        double rt, rp;
        march_part(P, j0 + j, R, sink, k0, k1, rt, rp);
        // non-negative doubles order as integers
        atomicMax(&resid_t[j0 + j], (unsigned long long)__double_as_longlong(rt));
        atomicMax(&resid_phi[j0 + j], (unsigned long long)__double_as_longlong(rp));
    } else {
        march_range(P, j0 + j, R, sink, k0, k1);
    }
}

// A block per (32 rays, segment of seg_len samples starting at an anchor multiple) of the rays [j0, j0 + npix), the
// samples by march_block. The FP64 stream also leaves the anchor residuals of its rays (the largest over the segments).
template <class T, class S>
__global__ void __launch_bounds__(32 * kMarchWarps, sizeof(T) == 4 ? 4 : 3)
k_stream_block(PlanView P, Spacetime st, long long j0, long long npix, long long npad, int seg_len, S* __restrict__ out,
               unsigned long long* __restrict__ resid_t, unsigned long long* __restrict__ resid_phi) {
    extern __shared__ __align__(16) unsigned char march_smem[];
    MarchShared<T>& shared = *reinterpret_cast<MarchShared<T>*>(march_smem);
    const int lane = threadIdx.x & 31;
    const bool live = blockIdx.x * 32LL + lane < npix;
    const long long j = live ? blockIdx.x * 32LL + lane : npix - 1;
    const int k0 = 1 + blockIdx.y * seg_len, k1 = min(st.N + 1, k0 + seg_len);
    const double temp = sqrt(1.0 - st.a * st.a);
    StreamSink<T, S> sink{out, npad, j, T(st.a), T(st.rh * (1 + 1e-3)), T(1.0 + temp), T(1.0 - temp), float(st.a / (2.0 * temp))};
    double rt, rp;
    march_block<sizeof(S) == 8>(P, st, j0 + j, live, k0, k1, shared, sink, rt, rp);
    if (sizeof(S) == 8 && threadIdx.x < 32 && live) {
        // non-negative doubles order as integers
        atomicMax(&resid_t[j0 + j], (unsigned long long)__double_as_longlong(rt));
        atomicMax(&resid_phi[j0 + j], (unsigned long long)__double_as_longlong(rp));
    }
}

// The adjoint's state of a sample: P before it (16), the coefficients (11), the step length: whole 16-byte words.
constexpr int kState = 28;

// A transport pass and its segmentation, as the reverse pass walks it too: work units of 32 consecutive sorted rays x
// one segment of the sample range x one frame x up to `ch` frequencies, the last rays first (the plunging rays
// near the centre of the screen, sorted last, carry most of the work).
struct TransportJob {
    long long npix, npad;            // rays and the stride of the plan, of the stream and of the output rows
    int nframes, nfreq, nseg, seg_len, nvc;
    long long nchunks;               // 32-ray groups
    double L;
    void* gstate = nullptr;          // the adjoint's state: kState values of T per (combination, sample, ray)
    unsigned char* gact = nullptr;   // and 1 where the sample has a step
    const int* kstop = nullptr;      // the first sample beyond the half-orbit cutoff (null: none)
    int ntot = 0, nkv = 0, run = 64, cap = 0, rows_shared = 1;
    long long j0 = 0;                // first ray of the launch (npix counts from it)
    int stage_test = 0;              // test hook: arm the table-staging barrier without the copy
    int ch = 1;                      // frequencies per work unit
};

}  // namespace ks
