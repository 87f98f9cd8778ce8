// ks_forward.cu -- the forward pass of the polarized renders: the sample stream (ks_mixed.cuh) and the transport
// over it (ks_transport.cuh), in FP32 or FP64, with the rules that size their launches.
#include <algorithm>
#include <cmath>

#include "../../include/kerrsplat_b200.h"
#include "ks_transfer.cuh"

static __constant__ ks::MomentCoeffs c_moments;

#include "ks_context.cuh"
#include "ks_transport.cuh"

using namespace ks;

int forward_init(const MomentCoeffs& mc) { return cudaMemcpyToSymbol(c_moments, &mc, sizeof mc) == cudaSuccess ? KS_OK : KS_ERR_DEVICE; }

// The FP32 sample stream of every ray (k_stream: the FP32 march, or the FP64 march under
// KS_MIXED_GEO64), [k][field][npad]. Each ray is marched as up to eight segments, each starting
// at an anchor (a multiple of M samples). At 256 x 256, N = 1024 that is 6.9 waves of 16 warps per
// SM instead of 3.5 with four segments (the render 22.04 against 22.34 ms).
static int stream_segments(const ks_context* c, int* len) {
    const int M = c->st.M, N = c->st.N;
    *len = std::max(M, (N / 8 + M - 1) / M * M);
    return (N + *len - 1) / *len;
}

// The stream kernel of (ray, segment) pairs: a block marching 32 rays together while there are few of them, a thread
// each once they fill the chip. Measured in us, block against thread: FP32 at 512 samples (8 segments) 32 x 32 rays
// 94 : 234, 64 x 64 200 : 252, 80 x 80 286 : 276, 128 x 128 647 : 574; at 128 samples (2 segments) 128 x 128 201 : 260,
// 192 x 192 394 : 343. FP64 at 101 x 93 rays x 384 samples, with its transport, 1337 : 1420.
template <class T, class S>
static int stream_kernel(ks_context* c, long long j0, long long npix, long long npad, S* out) {
    int len = 0;
    const int nseg = stream_segments(c, &len);
    auto* rt = c->resid_t.as<unsigned long long>();
    auto* rp = c->resid_phi.as<unsigned long long>();
    if (npix * nseg < (sizeof(S) == 8 ? 65536 : 49152)) {
        const int smem = int(sizeof(MarchShared<T>));
        KS_CUDA(c, cudaFuncSetAttribute(k_stream_block<T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        k_stream_block<T, S><<<dim3(nblocks(npix, 32), nseg), 32 * kMarchWarps, smem, c->stream>>>(plan_view(c), c->st, j0, npix, npad, len, out, rt, rp);
    } else {
        k_stream<T, S><<<nblocks(npix * nseg, 128), 128, 0, c->stream>>>(plan_view(c), c->st, j0, npix, npad, len, nseg, out, rt, rp);
    }
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// ... of the rays [j0, j0 + m), npad apart
static int mixed_stream(ks_context* c, long long j0, long long m, long long npad) {
    KS_CUDA(c, c->stream_buf.ensure(size_t(c->st.N) * SM_COUNT * npad * sizeof(float)));
    float* out = c->stream_buf.as<float>();
    return c->geo64 ? stream_kernel<double, float>(c, j0, m, npad, out) : stream_kernel<float, float>(c, j0, m, npad, out);
}

template <class T>
static int wind_stop(ks_context* c, int nmax, double slab, long long j0, long long m, long long npad, const T* stream) {
    KS_CUDA(c, c->kstop.ensure(size_t(c->npix) * sizeof(int)));
    k_wind_stop<T><<<nblocks(m), kBlock, 0, c->stream>>>(plan_view(c), j0, m, npad, stream, nmax, T(slab), c->kstop.as<int>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

int launch_stream(ks_context* c) { return mixed_stream(c, 0, c->npix, c->npad); }

int launch_wind_stop(ks_context* c, int nmax, double slab) { return wind_stop(c, nmax, slab, 0, c->npix, c->npad, c->stream_buf.as<float>()); }

// How a transport kernel of NT threads is shaped for a scene: samples per run, records per window, blocks per SM.
struct Shape {
    int run = 0, cap = 0, blocks = 0;
    bool rows_shared = true;
    size_t smem = 0;
};

// The most blocks of the kernel (up to its register budget, `maxb`) whose rows, masks and at least one record a
// thread fit in shared memory; then the longest run, and up to two records a thread. Rows that leave no room at
// all stay in global memory.
template <class T, int CH, int KM, int NT>
static Shape transport_shape(int ntot, int nkv, int seg_len, int maxb) {
    using SM = TransportSmem<T, CH, KM, NT>;
    constexpr int W = NT / 32;
    const size_t all = 227 * 1024;
    for (int shared = 1; shared >= 0; --shared)
        for (int b = maxb; b >= 1; --b)
            for (int run : {64, 32, 16}) {
                if (run > 16 && run / 2 >= seg_len) continue;   // a run longer than the segment
                if (run / W < 1) continue;
                const size_t budget = std::min<size_t>(all, size_t(228 * 1024) / b - 1024 - 64);
                const size_t fixed = SM::bytes(ntot, nkv, run, 0, shared != 0);
                const size_t per = SM::REC * sizeof(T) + 4;
                if (fixed + 32 * per > budget) continue;
                int cap = int(std::min<size_t>((budget - fixed) / per, 2 * NT)) / 32 * 32;
                cap = std::min(cap, run * 32);
                if (cap < (b > 1 ? std::min(NT, run * 32) : 32)) continue;   // a thinner window than the block is wide: rather fewer blocks
                Shape s;
                s.run = run; s.cap = cap; s.blocks = b; s.rows_shared = shared != 0;
                s.smem = SM::bytes(ntot, nkv, run, cap, shared != 0);
                return s;
            }
    return Shape{};
}

template <class T, int CH, int KM, int NT, int MINB>
static int run_transport(ks_context* c, TransportJob job, const Shape& sh, T* stream, T* seg_out, long long nout) {
    auto* kernel = k_transport<T, CH, KM, NT, MINB>;
    KS_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sh.smem)));
    job.run = sh.run; job.cap = sh.cap; job.rows_shared = sh.rows_shared ? 1 : 0;
    const long long total = job.nchunks * job.nseg * job.nframes * job.nvc;
    const long long grid = std::min<long long>(total, (long long)c->nsm * sh.blocks);
    const double* dt = c->combos.as<double>();
    KS_CUDA(c, cudaMemsetAsync(c->work.p, 0, sizeof(unsigned long long), c->stream));
    const bool timed = sizeof(T) == 4 && !c->capturing;   // ks_consume_stats
    if (timed) cudaEventRecord(c->evc0, c->stream);
    kernel<<<unsigned(grid), NT, sh.smem, c->stream>>>(plan_view(c), c->st, job, c->rows.as<T>(), dt, dt + job.nframes, stream,
                                                       c->work.as<unsigned long long>(), seg_out,
                                                       c->count_events ? c->counters.as<unsigned long long>() : nullptr, c->errflag.as<unsigned>());
    if (timed) {
        cudaEventRecord(c->evc1, c->stream);
        c->consume_timed = true;
    }
    c->launches++;
    c->kernel_launches++;
    KS_CUDA(c, cudaGetLastError());
    const long long nq = job.npix * (long long)job.nframes * job.nfreq;
    k_compose<T><<<nblocks(nq, 256), 256, 0, c->stream>>>(job, dt + job.nframes, seg_out, nout, c->out_sorted.as<double>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// The sample range in segments until there are some units per resident block (default 8, or the autotuner's
// choice), so that the most expensive unit is short; segments keep at least 16 samples.
static void segment(TransportJob& job, int N, long long blocks, int per_block) {
    const long long base = job.nchunks * job.nframes * job.nvc;
    int nseg = 1;
    while (base * nseg < per_block * blocks && (nseg * 2) * 16 <= N) nseg *= 2;
    job.seg_len = (N + nseg - 1) / nseg;
    job.nseg = (N + job.seg_len - 1) / job.seg_len;
}

template <class T, int KM>
static int build_rows(ks_context* c, int ntot, bool grad) {
    const long long total = ((long long)ntot * row_stride<T, KM>() + c->nkv + 3) / 4 * 4 + 4;
    KS_CUDA(c, c->rows.ensure(size_t(total) * sizeof(T)));
    k_rows<T, KM><<<nblocks(total, 256), 256, 0, c->stream>>>(ntot, c->nkv, total, c->tab.as<double>(), grad ? c->gtab.as<double>() : nullptr, c->rows.as<T>());
    c->launches++;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

static TransportJob transport_job(ks_context* c, int ntot, int nframes, int nfreq, int ch, double L, long long j0, long long npix, long long npad) {
    TransportJob job;
    job.npix = npix; job.npad = npad; job.j0 = j0;
    job.nframes = nframes; job.nfreq = nfreq; job.nvc = (nfreq + ch - 1) / ch;
    job.nchunks = (npix + 31) / 32;
    job.L = L; job.ntot = ntot; job.nkv = c->nkv; job.ch = ch;
    job.stage_test = c->stage_test;
    return job;
}

// The rays [j0, j0 + m), npad apart in the stream and the state (the reverse pass's, if there is one).
template <int CH, int KM>
static int mixed_ch(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, long long j0, long long m, long long npad,
                    float* gstate, unsigned char* gact) {
    // one march per ray, shared by every frame and frequency
    int s = mixed_stream(c, j0, m, npad);
    if (s || (s = build_rows<float, KM>(c, ntot, gstate != nullptr))) return s;
    TransportJob job = transport_job(c, ntot, nframes, nfreq, CH, L, j0, m, npad);
    if (nmax >= 0) {
        if ((s = wind_stop(c, nmax, slab, j0, m, npad, c->stream_buf.as<float>()))) return s;
        job.kstop = c->kstop.as<int>();
    }
    constexpr int B128 = 4, B256 = 2;
    Shape s128 = transport_shape<float, CH, KM, 128>(ntot, c->nkv, c->st.N, B128), s256 = transport_shape<float, CH, KM, 256>(ntot, c->nkv, c->st.N, B256);
    // the largest table (splat constants and knots) a call may bring, by its frequencies (four or more as many as two); its
    // rows stay in global memory where a block's shared memory does not hold them
    constexpr int kBound = CH == 4 ? 2 : CH;
    if (((size_t)ntot * ST_COUNT + c->nkv) * sizeof(float) > 227 * 1024 - 4 * (5848 + 4096 * size_t(kBound))) s128.blocks = s256.blocks = 0;
    if (s128.blocks == 0 && s256.blocks == 0) return fail(c, KS_ERR_ARGUMENT, "too many splats for one launch (%d)", ntot);
    // the wider block where shared memory (a large table) holds more of its warps, or the autotuner's choice
    bool wide = s256.blocks * 8 > s128.blocks * 4;
    if (c->tune_nt == 256 && s256.blocks > 0) wide = true;
    if (c->tune_nt == 128 && s128.blocks > 0) wide = false;
    segment(job, c->st.N, (long long)c->nsm * (wide ? s256.blocks : s128.blocks), c->tune_units > 0 ? c->tune_units : 8);
    // runs no longer than a segment
    if (wide) s256 = transport_shape<float, CH, KM, 256>(ntot, c->nkv, job.seg_len, B256);
    else s128 = transport_shape<float, CH, KM, 128>(ntot, c->nkv, job.seg_len, B128);
    job.gstate = gstate;
    job.gact = gact;
    c->last_job = job;   // as the reverse pass walks it
    KS_CUDA(c, c->seg_out.ensure(size_t(nframes) * nfreq * job.nseg * m * 20 * sizeof(float)));
    KS_CUDA(c, c->work.ensure(2 * sizeof(unsigned long long)));   // the adjoint's two counters: no move under a captured render
    return wide ? run_transport<float, CH, KM, 256, B256>(c, job, s256, c->stream_buf.as<float>(), c->seg_out.as<float>(), c->npix)
                : run_transport<float, CH, KM, 128, B128>(c, job, s128, c->stream_buf.as<float>(), c->seg_out.as<float>(), c->npix);
}

// Up to four frequencies share a unit's march, tests and frames.
template <int KM>
static int mixed_km(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, long long j0, long long m, long long npad,
                    float* gstate, unsigned char* gact) {
    if (ntot > 32 * kMaxSplatWords) return fail(c, KS_ERR_ARGUMENT, "the mixed path takes at most %d splats (%d)", 32 * kMaxSplatWords, ntot);
    if (nfreq >= 4) return mixed_ch<4, KM>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, npad, gstate, gact);
    if (nfreq == 3) return mixed_ch<3, KM>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, npad, gstate, gact);
    if (nfreq == 2) return mixed_ch<2, KM>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, npad, gstate, gact);
    return mixed_ch<1, KM>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, npad, gstate, gact);
}

int launch_mixed(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, bool thermal_only) {
    return thermal_only ? mixed_km<1>(c, ntot, nframes, nfreq, L, nmax, slab, 0, c->npix, c->npad, nullptr, nullptr)
                        : mixed_km<7>(c, ntot, nframes, nfreq, L, nmax, slab, 0, c->npix, c->npad, nullptr, nullptr);
}

// FP64: the rays [j0, j0 + m), their stream and the transport over it; npad strides the stream and the state.
template <int KM>
static int plain_piece(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, long long j0, long long m, long long npad,
                       double* gstate, unsigned char* gact) {
    const int N = c->st.N;
    KS_CUDA(c, c->stream64.ensure(size_t(npad) * N * SM_COUNT * sizeof(double)));
    KS_CUDA(c, c->work.ensure(2 * sizeof(unsigned long long)));
    double* stream = c->stream64.as<double>();
    {
        int s = stream_kernel<double, double>(c, j0, m, npad, stream);
        if (s) return s;
    }
    TransportJob job = transport_job(c, ntot, nframes, nfreq, 1, L, j0, m, npad);
    if (nmax >= 0) {
        const int s = wind_stop(c, nmax, slab, j0, m, npad, stream);
        if (s) return s;
        job.kstop = c->kstop.as<int>();
    }
    constexpr int B = 2;
    Shape sh = transport_shape<double, 1, KM, 128>(ntot, c->nkv, N, B);
    if (sh.blocks == 0) return fail(c, KS_ERR_ARGUMENT, "too many splats for one launch (%d)", ntot);
    segment(job, N, (long long)c->nsm * sh.blocks, 8);
    sh = transport_shape<double, 1, KM, 128>(ntot, c->nkv, job.seg_len, B);
    job.gstate = gstate; job.gact = gact;
    if (gstate) c->last_job = job;
    KS_CUDA(c, c->seg_out64.ensure(size_t(nframes) * nfreq * job.nseg * m * 20 * sizeof(double)));
    return run_transport<double, 1, KM, 128, B>(c, job, sh, stream, c->seg_out64.as<double>(), c->npix);
}

static int clear_residuals(ks_context* c) {
    KS_CUDA(c, cudaMemsetAsync(c->resid_t.p, 0, size_t(c->npix) * sizeof(double), c->stream));
    KS_CUDA(c, cudaMemsetAsync(c->resid_phi.p, 0, size_t(c->npix) * sizeof(double), c->stream));
    return KS_OK;
}

long long smaller_piece(long long rays) { return std::max<long long>(32, (rays / 2 + 31) / 32 * 32); }

// The rays in pieces of at most 4 GB of stream and 4 GB of segment states (in one segment), halved until they fit.
template <int KM>
static int plain_km(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab) {
    int s = build_rows<double, KM>(c, ntot, false);
    if (s || (s = clear_residuals(c))) return s;
    const size_t per_ray = std::max(size_t(c->st.N) * SM_COUNT, size_t(nframes) * nfreq * 20) * sizeof(double);
    long long piece = std::min<long long>(c->npad, std::max<long long>(32, (long long)((size_t(4) << 30) / per_ray) / 32 * 32));
    for (long long j0 = 0; j0 < c->npix;) {
        s = plain_piece<KM>(c, ntot, nframes, nfreq, L, nmax, slab, j0, std::min(piece, c->npix - j0), piece, nullptr, nullptr);
        if (s == KS_ERR_OUT_OF_MEMORY && piece > 32) {
            c->stream64.release();
            c->seg_out64.release();
            piece = smaller_piece(piece);
            j0 = 0;
            continue;
        }
        if (s) return s;
        j0 += piece;
    }
    return KS_OK;
}

// Mixed: every ray. FP64: rays whose state (225 bytes a sample and combination) fits in 24 GB.
long long state_rays(const ks_context* c, bool plain, int nframes, int nfreq) {
    if (!plain) return c->npad;
    const size_t per_ray = size_t(nframes) * nfreq * c->st.N * (kState * sizeof(double) + 1);
    return std::min<long long>(c->npad, std::max<long long>(32, (long long)((size_t(24) << 30) / per_ray) / 32 * 32));
}

int launch_state(ks_context* c, bool plain, int ntot, int nframes, int nfreq, double L, int nmax, double slab, long long j0, long long m, long long rays) {
    const size_t rows = size_t(nframes) * nfreq * c->st.N * rays;
    KS_CUDA(c, c->adj_state.ensure(rows * kState * (plain ? sizeof(double) : sizeof(float))));
    KS_CUDA(c, c->adj_act.ensure(rows));
    KS_CUDA(c, cudaMemsetAsync(c->adj_act.p, 0, rows, c->stream));
    if (!plain)
        return mixed_km<1>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, rays, c->adj_state.as<float>(), c->adj_act.as<unsigned char>());
    int s = build_rows<double, 1>(c, ntot, true);
    if (s || (j0 == 0 && (s = clear_residuals(c)))) return s;
    return plain_piece<1>(c, ntot, nframes, nfreq, L, nmax, slab, j0, m, rays, c->adj_state.as<double>(), c->adj_act.as<unsigned char>());
}

void release_state(ks_context* c) {
    for (DevBuf* d : {&c->adj_state, &c->adj_act, &c->adj_bnd, &c->adj_unit, &c->adj_part, &c->stream64, &c->seg_out64, &c->seg_out}) d->release();
}

int launch_plain(ks_context* c, int ntot, int nframes, int nfreq, double L, int nmax, double slab, bool thermal_only) {
    return thermal_only ? plain_km<1>(c, ntot, nframes, nfreq, L, nmax, slab) : plain_km<7>(c, ntot, nframes, nfreq, L, nmax, slab);
}
