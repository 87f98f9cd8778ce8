// ks_reverse.cu -- the reverse pass (ks_reverse.cuh): its launches and the reduction into parameter rows.
#include <algorithm>

#include "../../include/kerrsplat_b200.h"
#include "ks_transfer.cuh"

static __constant__ ks::MomentCoeffs c_moments;

#include "ks_context.cuh"
#include "ks_reverse.cuh"

using namespace ks;

int reverse_init(const MomentCoeffs& mc) { return cudaMemcpyToSymbol(c_moments, &mc, sizeof mc) == cudaSuccess ? KS_OK : KS_ERR_DEVICE; }

template <class T, int CH, int NT, int MINB>
static int reverse_ch(ks_context* c, int ntot, int nmax, bool add) {
    using SM = ReverseSmem<T, CH, NT>;
    constexpr bool plain = sizeof(T) == 8;
    TransportJob job = c->last_job;
    job.kstop = nmax >= 0 ? c->kstop.as<int>() : nullptr;
    // as many blocks as fit (registers hold MINB) with a full window each; the longest run, then the most records; rows
    // that leave no room stay in global memory
    const int nw = (ntot + 31) / 32;
    size_t smem = 0;
    for (int shared = 1; shared >= 0 && !smem; --shared)
        for (int b = MINB; b >= 1 && !smem; --b)
            for (int run : {64, 32, 16}) {
                if (run > 16 && run / 2 >= job.seg_len) continue;
                const size_t budget = std::min<size_t>(227 * 1024, size_t(228 * 1024) / b - 1024 - 64);
                int cap = std::min(2 * NT, run * 32);
                while (cap >= 32 && SM::bytes(ntot, run, cap, shared != 0) > budget) cap -= 32;
                if (cap < (b > 1 ? std::min(NT, run * 32) : 32)) continue;
                if (run > 16 && b > 1 && size_t(run) * 32 * nw * 4 > budget / 3) continue;   // masks of a large table: rather a shorter run
                job.run = run; job.cap = cap; job.rows_shared = shared; smem = SM::bytes(ntot, run, cap, shared != 0);
                break;
            }
    if (!smem) return fail(c, KS_ERR_ARGUMENT, "too many splats for the %s adjoint (%d)", plain ? "FP64" : "mixed", ntot);
    auto* kernel = k_reverse<T, CH, NT, MINB>;
    KS_CUDA(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int per_sm = 0;
    KS_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, NT, smem));
    const double* dt = c->combos.as<double>();
    const double* dn = dt + job.nframes;
    const long long ncombo = (long long)job.nframes * job.nfreq, total = job.nchunks * job.nseg * job.nframes * job.nvc;
    const T* seg_out = plain ? c->seg_out64.as<T>() : c->seg_out.as<T>();
    const T* stream = plain ? c->stream64.as<T>() : c->stream_buf.as<T>();
    KS_CUDA(c, c->adj_bnd.ensure(size_t(ncombo) * job.nseg * 8 * job.npix * sizeof(T)));
    k_adj_bounds<T><<<nblocks(job.npix * ncombo, 256), 256, 0, c->stream>>>(job, dn, seg_out, c->seeds.as<double>(), c->npix, c->adj_bnd.as<T>());
    const long long gsz = (long long)ntot * PS_COUNT;
    KS_CUDA(c, c->adj_unit.ensure(size_t(total) * gsz * sizeof(T)));
    KS_CUDA(c, c->work.ensure(2 * sizeof(unsigned long long)));
    KS_CUDA(c, cudaMemsetAsync(c->work.p, 0, 2 * sizeof(unsigned long long), c->stream));
    const long long grid = std::min<long long>(total, (long long)c->nsm * std::max(per_sm, 1));
    kernel<<<unsigned(grid), NT, smem, c->stream>>>(plan_view(c), c->st, job, c->rows.as<T>(), dt, dn, stream, c->adj_bnd.as<T>(),
                                                    c->work.as<unsigned long long>(), c->adj_unit.as<T>(), c->errflag.as<unsigned>());
    const int per_chunk = 256;
    const int nchunks = int((total + per_chunk - 1) / per_chunk);
    KS_CUDA(c, c->adj_part.ensure(size_t(nchunks) * gsz * sizeof(double)));
    k_unit_reduce1<T><<<dim3(nblocks(gsz, 128), nchunks), 128, 0, c->stream>>>(c->adj_unit.as<T>(), total, gsz, per_chunk, c->adj_part.as<double>());
    k_reverse_rows<<<ntot, 32, 0, c->stream>>>(c->adj_part.as<double>(), nchunks, ntot, c->tab.as<double>(), c->gtab.as<double>(), add ? 1 : 0,
                                               c->dgrad.as<double>());
    c->launches += 4;
    c->adjoint_launches += 4;
    KS_CUDA(c, cudaGetLastError());
    return KS_OK;
}

// The reverse pass groups frequencies as the forward pass did.
int launch_reverse(ks_context* c, int ntot, int nmax, bool plain, bool add) {
    if (plain) return reverse_ch<double, 1, 128, 2>(c, ntot, nmax, add);
    if (ntot > 32 * kMaxSplatWords) return fail(c, KS_ERR_ARGUMENT, "the mixed adjoint takes at most %d splats (%d)", 32 * kMaxSplatWords, ntot);
    switch (c->last_job.ch) {
        case 4: return reverse_ch<float, 4, 128, 3>(c, ntot, nmax, add);
        case 3: return reverse_ch<float, 3, 128, 3>(c, ntot, nmax, add);
        case 2: return reverse_ch<float, 2, 128, 3>(c, ntot, nmax, add);
        default: return reverse_ch<float, 1, 128, 3>(c, ntot, nmax, add);
    }
}
