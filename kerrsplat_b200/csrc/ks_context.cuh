// ks_context.cuh -- the library's context (the device-side GeodesicCache of cache.jl:85-125) and the helpers that
// its translation units share.
#pragma once
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "../../include/kerrsplat_b200.h"
#include "ks_mixed.cuh"

constexpr int kBlock = 128;

struct DevBuf {
    void* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;   // one owner per allocation
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    cudaError_t ensure(size_t bytes) {
        if (bytes <= n) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr; n = 0;
        cudaError_t e = cudaMalloc(&p, bytes);
        if (e == cudaSuccess) n = bytes;
        return e;
    }
    void release() { if (p) cudaFree(p); p = nullptr; n = 0; }
    void swap(DevBuf& o) { std::swap(p, o.p); std::swap(n, o.n); }
    template <class U> U* as() const { return reinterpret_cast<U*>(p); }
};

struct ks_context {
    int device = 0, nsm = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    long long npix = 0, npad = 0;
    int nalpha = 0, nbeta = 0;
    bool regenerated = false;
    ks::Spacetime st{};
    DevBuf alpha, beta, key, key2, idx, perm, plan, nanch, aoff, anchors, resid_t, resid_phi, scratch;
    DevBuf tab, combos, out_sorted, stage_in, stage_out, counters, seg_out, work, stream_buf;
    DevBuf inv_perm, dft_tu, dft_tv, dft_a, dft_t, dft_c, dft_s, dft_in[8], dft_partial;
    // adjoint: gradient table, cutoffs, the gradient, seeds, chi^2 partials; per-sample states, activity, segment bounds,
    // unit partials
    DevBuf gtab, kstop, dgrad, seeds, chi_part, chi_val, dstage;
    DevBuf adj_state, adj_act, adj_bnd, adj_unit, adj_part, jvp_tab, jvp_in, jvp_out, jvp_part, st_buf;
    DevBuf rows;      // the transport's splat rows and knot array (FP32 or FP64)
    DevBuf thin_part;             // the thin image's pieces (sized by regenerate)
    DevBuf stream64, seg_out64;   // the FP64 render's stream and segment states
    DevBuf errflag;   // set by a kernel whose bounded wait gave up
    cudaGraph_t graph = nullptr;          // ks_render_graph_capture: one mixed render of device-resident sets
    cudaGraphExec_t graph_exec = nullptr;
    cudaGraph_t cgraph = nullptr;         // ks_chi2_gradient_graph_capture: one mixed chi^2 + gradient evaluation
    cudaGraphExec_t cgraph_exec = nullptr;
    std::vector<void*> cgraph_bufs;
    // what a captured graph reads of its own call: the splat table with the knots, the times and the frequencies
    DevBuf graph_tab, graph_combos, cgraph_tab, cgraph_combos;
    bool capturing = false;               // inside that capture: no timing events
    int stage_test = 0;                   // ks_set_stage_test
    std::vector<void*> graph_bufs;        // the buffers the graph uses, as captured (a replay checks them)
    
    int tune_nt = 0, tune_units = 0;        // the autotuner's choice for the mixed forward (0: the default)
    int nkv = 0;                            // knot values after the splat table in `tab`
    ks::TransportJob last_job{};            // the last forward pass with an adjoint's state
    long long state_piece = 0;              // rays whose state the last gradient held at a time
    double adjoint_ms = 0.0;
    long long adjoint_launches = 0;
    bool count_events = false;
    int tensor_path = 0;  // 3xTF32 GEMMs: 0 tcgen05 (k_gemm_tc), 1 mma.sync (k_gemm_3xtf32); ks_set_tensor_path
    bool geo64 = false;   // mixed path: the FP64 march feeds the FP32 transport (KS_MIXED_GEO64) instead of the FP32 march
    long long total_anchors = 0;
    int max_nanch = 0;
    long long ranges[6] = {0, 0, 0, 0, 0, 0};
    // timing of the render kernels (CUDA events on the context stream)
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t evc0 = nullptr, evc1 = nullptr;   // around k_transport (the mixed path's dominant kernel)
    cudaEvent_t evg0 = nullptr, evg1 = nullptr;   // around each 3xTF32 GEMM (outside graph captures)
    double gemm_ms = 0.0, gemm_flops = 0.0;       // ks_gemm_stats: device time and tensor-core flops (3 x 2 M N K)
    long long gemm_launches = 0;
    bool consume_timed = false;
    double consume_ms = 0.0;
    long long consume_launches = 0;
    double kernel_ms = 0.0;
    long long kernel_launches = 0;
    long long launches = 0;
};

inline int fail(ks_context* c, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    return code;
}

inline int cuda_fail(ks_context* c, cudaError_t e, const char* what) {
    cudaGetLastError();   // reported here: the next call (of any context) checks its own launches
    if (e == cudaErrorMemoryAllocation) return fail(c, KS_ERR_OUT_OF_MEMORY, "%s: %s", what, cudaGetErrorString(e));
    return fail(c, KS_ERR_DEVICE, "%s: %s", what, cudaGetErrorString(e));
}

#define KS_CUDA(ctx, call)                                            \
    do {                                                              \
        cudaError_t e_ = (call);                                      \
        if (e_ != cudaSuccess) return cuda_fail((ctx), e_, #call);    \
    } while (0)

inline bool is_device_ptr(const void* p) {
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Make `src` (host or device, `bytes`) available on the device: returns the device pointer.
inline int stage_in(ks_context* c, DevBuf& buf, const void* src, size_t bytes, const void** dev) {
    if (is_device_ptr(src)) { *dev = src; return KS_OK; }
    KS_CUDA(c, buf.ensure(bytes));
    KS_CUDA(c, cudaMemcpyAsync(buf.p, src, bytes, cudaMemcpyHostToDevice, c->stream));
    *dev = buf.p;
    return KS_OK;
}

inline unsigned nblocks(long long n, int b = kBlock) { return unsigned((n + b - 1) / b); }

inline ks::PlanView plan_view(ks_context* c) {
    ks::PlanView P;
    P.f = c->plan.as<double>(); P.npad = c->npad; P.anchors = c->anchors.as<double>(); P.anchor_off = c->aoff.as<long long>();
    return P;
}


// ---- the forward pass (ks_forward.cu) -------------------------------------------------------------------

// Constants of the forward kernels on the current device.
int forward_init(const ks::MomentCoeffs& mc);
// The FP32 sample stream of every ray.
int launch_stream(ks_context* c);
// The half-orbit cutoff of every ray on the FP32 stream, into c->kstop.
int launch_wind_stop(ks_context* c, int nmax, double slab);
// The render into c->out_sorted from the tables that build_tables left: FP32 transport over the FP32 stream, or
// FP64 throughout. The times, then the frequencies, lie in c->combos.
int launch_mixed(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, bool thermal_only);
int launch_plain(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, bool thermal_only);
// The pass over the rays [j0, j0 + m) of a thermal scene with the reverse pass's state, sized for `rays` rays: at most
// state_rays. KS_ERR_OUT_OF_MEMORY: release_state, then again with a smaller_piece.
long long state_rays(const ks_context* c, bool plain, int nframes, int nfreq);
int launch_state(ks_context* c, bool plain, int ntot, int nframes, int nfreq, double L, int nmax, double slab, long long j0, long long m, long long rays);
void release_state(ks_context* c);
long long smaller_piece(long long rays);

// ---- the mixed reverse pass (ks_reverse.cu) --------------------------------------------------------------

int reverse_init(const ks::MomentCoeffs& mc);
// The gradient into c->dgrad (added to it with `add`) from the state of the last forward pass with one, FP32 or FP64
// (`plain`), and the seeds in c->seeds.
int launch_reverse(ks_context* c, int ntot, int nmax, bool plain, bool add);
