// pdf_resident.cu -- the resident forward kernel: sim, forward mark, prune
// and merge of a netlist that fits on chip.
//
// What bounds such a walk is its chain of levels, not bytes: the staged
// kernel (forward_cta) pays a piece descriptor, a TMA copy and a barrier of a
// whole CTA for every level, about 1 us each, on levels of a few dozen gates.
// Here a CTA brings the whole netlist into shared memory with one bulk copy
// (16-byte records and 16-bit edges, the image that build_resident lays out),
// keeps every gate's V, T and M words there, and then takes a level in one
// shared-memory round trip and one barrier.  A thread is one (gate, word) of
// the block of BW words: narrow levels still give BW times their gates in
// threads.  Only the surviving marks (for the cover) and the first-detecting
// pairs leave the SM.  A CTA grades `per` column blocks one after another, so
// the image is read once per CTA.
//
// Measured (B200, kernel, us): a 20,000-gate circuit's 523 needed gates at
// 32,768 pairs 45 -> 22; a 1M-gate circuit's at 65,536 pairs 125 -> 59; 7,000
// gates that all switch at 3,776 pairs 92 -> 28.  The first and the last wait at
// the levels' barriers most (7 and 14 warps of an issue; memory 1 to 2), issue 42 %
// and 18 % active, DRAM at 1 % of its peak.
//
// With planes (OUT) it walks every gate that is not constant, all levels, and
// stores codes as it finds them (20,000 gates x 32,768 pairs, 3,400 of them
// not constant: 59 us beside a fill pass of 42; the staged walk of all gates
// took 277, the whole call 370 -> 188).  Blocks of 4 words make a row's piece
// 16 bytes; the other half of its sector follows with the CTA's next block.
#include "pdf_kernels.cuh"
#include "pdf_ptx.cuh"

#include <algorithm>

namespace {

template <int BW, int SEM, int OUT>
__device__ __forceinline__ void resident_cta(const FwdArgs &a, const uint32_t cta) {
    constexpr bool FIX = SEM >= 2;
    constexpr uint32_t kGroup = BW == 32 ? 0xFFFFFFFFu : (1u << BW) - 1u;
    extern __shared__ __align__(128) unsigned char smraw[];
    const uint4 *rec = reinterpret_cast<const uint4 *>(smraw);
    const uint16_t *edge = reinterpret_cast<const uint16_t *>(smraw + a.off_edge);
    const uint2 *lvl = reinterpret_cast<const uint2 *>(smraw + a.off_fid);  // first gate, observable gates
    // the caller's gate ids (in the image where they fit)
    const uint32_t *ids = a.image_ids ? reinterpret_cast<const uint32_t *>(lvl + a.c.n_levels + 1) : nullptr;
    const auto net = [&](uint32_t g) { return ids ? ids[g] : net_id(a.c, g); };
    uint2 *vt = reinterpret_cast<uint2 *>(smraw + a.off_ring);              // [gate][BW] V, T
    uint32_t *ms = reinterpret_cast<uint32_t *>(smraw + a.off_rec);         // [gate][BW] marks
    uint32_t *bm = reinterpret_cast<uint32_t *>(smraw + a.off_bm);
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smraw + a.off_mbar);
    // a gate's words of the caller's planes (what is asked for in full is
    // written as it is found; stores do not hold the level chain up)
    const auto put = [&](uint32_t g, uint32_t w, uint32_t V, uint32_t T) {
        const uint32_t id = net(g);
        if (id == kEmpty) return;  // a constant that stands for the fan-ins left out
        a.out_v[(size_t)id * a.out_ld + w] = V;
        a.out_t[(size_t)id * a.out_ld + w] = T;
    };
    __shared__ uint32_t s_reach, s_top, s_max;
    const uint32_t tid = threadIdx.x, NT = blockDim.x, lane = tid & 31;
    const uint32_t L = a.c.n_levels;
    const uint32_t b0 = cta * a.per, b1 = min(a.n_blocks, b0 + a.per);
    if (tid == 0) {
        mbar_init(mbar, 1);
        fence_mbar_init();
        mbar_expect_tx(mbar, a.image_bytes);
        bulk_g2s(smraw, a.image, a.image_bytes, mbar);
    }
    // The image is the circuit's own; the rest follows what is before this
    // launch in the stream.  With planes that is k_fill_planes, which itself
    // followed everything else and writes other rows of V and T: only the marks
    // wait for it.
    if (OUT == RES_LEAN) grid_wait();
    // the batch's cover state (the cover kernels run after this one)
    if (a.active) {
        for (uint32_t w = b0 * BW + tid; w < min(a.W, b1 * BW); w += NT) a.active[w] = 0;
        if (b1 == a.n_blocks && tid == 0) a.active[a.W] = 0;
    }
    if (a.acc && cta == 0 && tid == 0) {
        a.acc->batch_lo = 0;
        a.acc->batch_hi = 0;
        a.acc->batch_flags = 0;
        a.acc->done = 0;
        a.acc->n_over = 0;
        a.acc->done_over = 0;
    }
    __syncthreads();
    if (__syncthreads_or(!mbar_wait(mbar, 0, a.wait_polls))) {
        // no CTA leaves with a copy in flight; its blocks are published empty
        (void)mbar_wait(mbar, 0);
        for (uint32_t blk = b0; OUT != RES_SIM && blk < b1; blk++) {
            for (uint32_t q = tid; q < a.bm_words; q += NT) a.nzb[(size_t)blk * a.bm_words + q] = 0;
            if (tid == 0) a.blk_maxlvl[blk] = 0;
        }
        if (tid == 0) atomicOr(a.err, kErrTimeout);
        grid_wait();
        return;
    }
    const uint32_t j = tid & (BW - 1);         // this thread's word of the block (NT is a multiple of BW)
    const uint32_t step = NT / BW;             // gates per pass
    for (uint32_t blk = b0; blk < b1; blk++) {
        const uint32_t w = blk * BW + j;
        const uint32_t wm = w + 1 < a.W ? 0xFFFFFFFFu
                                        : (w + 1 == a.W ? ((a.n_pairs & 31) ? (1u << (a.n_pairs & 31)) - 1u : 0xFFFFFFFFu)
                                                        : 0u);
        for (uint32_t q = tid; q < a.bm_words; q += NT) bm[q] = 0;
        if (tid == 0) {
            s_reach = 0;
            s_top = 0;
            s_max = 0;
        }
        // ---- level 0: inputs (simkernel.cuh:112-125) and the constants; four
        // input words in flight per thread
        uint32_t my_reach = 0;
        bool any = false;
        const uint32_t n0 = lvl[1].x;
        __syncthreads();
        for (uint32_t g0 = tid / BW; g0 < n0; g0 += 4 * step) {
            uint32_t h[4], v[4], t[4], rw[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t g = g0 + u * step;
                h[u] = v[u] = t[u] = 0;
                if (g >= n0) continue;
                const uint4 r = rec[g];
                h[u] = r.x;
                rw[u] = r.w;
                if ((r.x & RF_INPT) && wm) {
                    v[u] = __ldg(a.pi_v + (size_t)r.y * a.pi_ld + w);
                    t[u] = __ldg(a.pi_t + (size_t)r.y * a.pi_ld + w);
                } else if (r.x & RF_OINV) {
                    v[u] = 0xFFFFFFFFu;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t g = g0 + u * step;
                if (g >= n0) continue;
                const uint32_t T = t[u] & wm, M = OUT == RES_SIM ? 0u : T & flagmask(h[u], RF_MARKF0);
                vt[g * BW + j] = make_uint2(v[u] & wm, T);
                if (OUT != RES_LEAN && wm) put(g, w, v[u] & wm, T);
                if (OUT == RES_SIM) continue;
                ms[g * BW + j] = M;
                if (M) {
                    any = true;
                    my_reach = max(my_reach, rw[u] >> 16);
                }
            }
        }
        // ---- the levels above (simkernel.cuh:126-149, markkernel.cuh:226-267),
        // until no marked gate carries further
        for (uint32_t l = 0;; l++) {
            if (l) {
                any = false;
                const uint32_t g1 = lvl[l + 1].x;
                for (uint32_t g = lvl[l].x + tid / BW; g < g1; g += step) {
                    const uint4 r = rec[g];
                    const uint32_t h = r.x, nfi = (h >> 8) & 0xFFu, nfold = hdr_nfold(h), eo = r.w & 0xFFFFu;
                    const auto fan = [&](uint32_t q) -> uint32_t {
                        return q < 4 ? ((q < 2 ? r.y : r.z) >> (16 * (q & 1))) & 0xFFFFu : edge[eo + q];
                    };
                    uint2 f[kInlineFanins];  // fan-ins 0..3
#pragma unroll
                    for (int q = 0; q < kInlineFanins; q++)
                        if ((uint32_t)q < nfi) f[q] = vt[fan(q) * BW + j];
                    uint32_t V, T, v1, M = 0;
                    eval_first(h, f[0].x, f[0].y, V, v1);
#pragma unroll
                    for (int q = 1; q < kInlineFanins; q++)
                        if ((uint32_t)q <= nfold) eval_fold<FIX>(h, V, v1, f[q].x, f[q].y);
                    for (uint32_t q = kInlineFanins; q <= nfold; q++) {
                        const uint2 x = vt[fan(q) * BW + j];
                        eval_fold<FIX>(h, V, v1, x.x, x.y);
                    }
                    eval_finish<FIX>(h, V, v1, T);
                    V &= wm;
                    T &= wm;
                    vt[g * BW + j] = make_uint2(V, T);
                    if (OUT != RES_LEAN && wm) put(g, w, V, T);
                    if (OUT == RES_SIM) continue;
                    if ((h & RF_MARKF0) && T) {
                        M = T & ms[fan(0) * BW + j];
                        if ((h & RF_SENS) && M) {
                            SensAcc s;
                            sens_init(s);
                            const bool or_like = (h & RF_IM) != 0;
#pragma unroll
                            for (int q = 0; q < kInlineFanins; q++)
                                if ((uint32_t)q < nfi) sens_step<SEM & 1>(s, or_like, f[q].x, f[q].y);
                            for (uint32_t q = kInlineFanins; q < nfi; q++) {
                                const uint2 x = vt[fan(q) * BW + j];
                                sens_step<SEM & 1>(s, or_like, x.x, x.y);
                            }
                            M &= sens_result<SEM & 1>(s);
                        }
                    } else if (FIX && (h & RF_MANY) && T) {
                        const uint32_t mor = flagmask(h, RF_IM), mxor = flagmask(h, RF_XOR), mand = ~(mor | mxor);
                        SensAcc s;
                        sens_init(s);
#pragma unroll
                        for (int q = 0; q < kInlineFanins; q++)
                            if ((uint32_t)q < nfi)
                                sens_step_fixed<SEM == PDF_MARK_FIXED_NONROBUST>(s, mand, mor, mxor, f[q].x, f[q].y,
                                                                                 ms[fan(q) * BW + j]);
                        for (uint32_t q = kInlineFanins; q < nfi; q++) {
                            const uint2 x = vt[fan(q) * BW + j];
                            sens_step_fixed<SEM == PDF_MARK_FIXED_NONROBUST>(s, mand, mor, mxor, x.x, x.y,
                                                                             ms[fan(q) * BW + j]);
                        }
                        M = T & sens_result<SEM == PDF_MARK_FIXED_NONROBUST>(s);
                    }
                    ms[g * BW + j] = M;
                    if (M) {
                        any = true;
                        my_reach = max(my_reach, r.w >> 16);
                    }
                }
            }
            if (__any_sync(0xFFFFFFFFu, any)) {
                const uint32_t wr = __reduce_max_sync(0xFFFFFFFFu, my_reach);
                if (lane == 0) {
                    s_top = l + 1;  // every warp that stores in level l stores this
                    if (wr > l) atomicMax(&s_reach, wr);
                }
            }
            __syncthreads();
            // s_reach grows past l only in threads that go on, so all decide alike
            if (l + 1 >= L || (OUT == RES_LEAN && s_reach <= l)) break;
        }
        if (OUT == RES_SIM) continue;
        if (OUT == RES_PLANES) grid_wait();
        // ---- prune (markkernel.cuh:271-293) and merge (mergekernel.cuh:116-198),
        // levels descending: a gate's mark is final once its fan-outs' are.
        // Gates from level s_top on hold no mark, and past the last level walked
        // their words are not this block's.
        const uint32_t g_top = lvl[s_top].x;
        for (int l = (int)s_top - 1; l >= 0; l--) {
            const uint2 lv = lvl[l];
            for (uint32_t k0 = 0; k0 < lv.y; k0 += step) {
                const uint32_t k = k0 + tid / BW, g = lv.x + k;
                uint32_t nm = 0;
                if (k < lv.y) {
                    const uint32_t m = ms[g * BW + j];
                    if (m) {
                        const uint4 r = rec[g];
                        uint32_t keep = (r.x & (1u << 4)) ? 0xFFFFFFFFu : 0u;
                        if (!keep) {
                            const uint32_t nfi = (r.x >> 8) & 0xFFu, e1 = rec[g + 1].w & 0xFFFFu;
                            for (uint32_t e = (r.w & 0xFFFFu) + (nfi > kInlineFanins ? nfi : 0); e < e1; e++)
                                if (edge[e] < g_top) keep |= ms[(uint32_t)edge[e] * BW + j];
                        }
                        nm = m & keep;
                        if (nm != m) ms[g * BW + j] = nm;
                    }
                }
                const uint32_t z = __ballot_sync(0xFFFFFFFFu, nm != 0);
                if (!z) continue;  // the same on every lane
                const uint32_t sh = lane & ~(uint32_t)(BW - 1), below = (1u << j) - 1u;
                const uint32_t V = nm ? vt[g * BW + j].x : 0u, x = nm & ~V, y = nm & V;
                const uint32_t bx = (__ballot_sync(0xFFFFFFFFu, x != 0) >> sh) & kGroup;
                const uint32_t by = (__ballot_sync(0xFFFFFFFFu, y != 0) >> sh) & kGroup;
                if ((z >> sh) & kGroup) {  // the gate keeps a mark in the block
                    a.M[(size_t)g * a.ld + w] = nm;  // (rows hold whole blocks)
                    if (OUT == RES_PLANES && nm) a.out_m[(size_t)net(g) * a.out_ld + w] = nm;
                    if (j == 0) atomicOr(bm + (g >> 5), 1u << (g & 31));
                    // the lowest word of each direction holds its first pair
                    if (x && !(bx & below)) atomicMin(a.first_x + net(g), a.pair_base + w * 32 + (__ffs(x) - 1));
                    if (y && !(by & below)) atomicMin(a.first_y + net(g), a.pair_base + w * 32 + (__ffs(y) - 1));
                }
                if (lane == 0) atomicMax(&s_max, (uint32_t)l + 1);
            }
            __syncthreads();
        }
        // the bitmap of surviving marks, for the cover kernels
        for (uint32_t q = tid; q < a.bm_words; q += NT) a.nzb[(size_t)blk * a.bm_words + q] = bm[q];
        if (tid == 0) a.blk_maxlvl[blk] = s_max;
        __syncthreads();
    }
}

template <int BW, int SEM, int OUT>
__global__ void __launch_bounds__(kResidentThreads, kResidentCtas) k_resident(const FwdArgs a) {
    grid_trigger();
    resident_cta<BW, SEM, OUT>(a, blockIdx.x);
    grid_wait();
}

// Rows that a resident walk with planes leaves out, a warp per row: bound by
// the stores (20,000 gates, of which 3,400 are not constant, x 32,768 pairs:
// 220 MB in 42 us).  VEC: rows start on 16 bytes.  A CTA per SM, so that the
// resident walk's fit beside them.
constexpr uint32_t kFillThreads = 512;
template <bool VEC>
__global__ void __launch_bounds__(kFillThreads) k_fill_planes(const int8_t *value, uint32_t G, uint32_t W, uint32_t last,
                                                     uint32_t *v, uint32_t *t, uint32_t *m, uint64_t ld) {
    grid_trigger();  // k_resident computes beside the stores
    const uint32_t lane = threadIdx.x & 31;
    const auto fill = [&](uint32_t *p, uint32_t x) {
        const uint32_t n4 = VEC ? (W - 1) / 4 : 0;  // the last word, which may hold fewer pairs, is not among them
        if constexpr (VEC)
            for (uint32_t q = lane; q < n4; q += 32) __stcs(reinterpret_cast<uint4 *>(p) + q, make_uint4(x, x, x, x));
        for (uint32_t w = 4 * n4 + lane; w < W; w += 32) __stcs(p + w, w + 1 == W ? x & last : x);
    };
    constexpr uint32_t kWarps = kFillThreads / 32;
    for (uint32_t g = blockIdx.x * kWarps + threadIdx.x / 32; g < G; g += gridDim.x * kWarps) {
        const int c = value[g];
        if (m) fill(m + (size_t)g * ld, 0u);
        if (c < 0) continue;
        fill(v + (size_t)g * ld, c ? 0xFFFFFFFFu : 0u);
        fill(t + (size_t)g * ld, 0u);
    }
}

// The circuits of a batch whose netlists fit on chip.
template <int BW, int SEM>
__global__ void __launch_bounds__(kResidentThreads, kResidentCtas)
    k_batch_resident(const FwdArgs *args, const uint32_t *bpref, uint32_t n, BatchCtl *ctl, uint32_t blk0) {
    __shared__ FwdArgs s_a;
    __shared__ uint32_t s_blk;
    if (threadIdx.x == 0) {
        const uint32_t gb = blk0 + blockIdx.x;
        const uint32_t ci = prefix_find(bpref, n, gb);
        s_a = args[ci];
        s_blk = gb - __ldg(bpref + ci);
        if (gb == 0) batch_begin(ctl);
    }
    __syncthreads();
    resident_cta<BW, SEM, RES_LEAN>(s_a, s_blk);
}

template <int BW, int SEM, int OUT>
cudaError_t launch_out(const FwdArgs &a, uint32_t ctas, uint32_t threads, size_t smem, cudaStream_t st) {
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(k_resident<BW, SEM, OUT>), smem);
    if (e != cudaSuccess) return e;
    if (!ctas || threads % 32 || threads > kResidentThreads) return cudaErrorInvalidValue;
    return launch_next(k_resident<BW, SEM, OUT>, ctas, threads, smem, st, a);
}
template <int BW, int SEM>
cudaError_t launch_t(const FwdArgs &a, int out, uint32_t ctas, uint32_t threads, size_t smem, cudaStream_t st) {
    switch (out) {
        case RES_LEAN: return launch_out<BW, SEM, RES_LEAN>(a, ctas, threads, smem, st);
        case RES_PLANES: return launch_out<BW, SEM, RES_PLANES>(a, ctas, threads, smem, st);
        // the values depend on the marks' table only through n-input XOR
        default: return launch_out<BW, SEM & 2, RES_SIM>(a, ctas, threads, smem, st);
    }
}
template <int BW, int SEM>
cudaError_t launch_batch_t(const BatchLaunch &b, const BatchClass &c, cudaStream_t st) {
    k_batch_resident<BW, SEM><<<c.blocks, c.threads, c.smem, st>>>(b.fargs, b.bpref, b.n, b.ctl, c.blk0);
    return cudaGetLastError();
}

// f<BW, SEM>() for run-time values.
#define PDF_RES_SEM(BW, F, ...)                      \
    switch (sem) {                                   \
        case 0: return F<BW, 0>(__VA_ARGS__);        \
        case 1: return F<BW, 1>(__VA_ARGS__);        \
        case 2: return F<BW, 2>(__VA_ARGS__);        \
        case 3: return F<BW, 3>(__VA_ARGS__);        \
        default: return cudaErrorInvalidValue;       \
    }
#define PDF_RES(F, ...)                              \
    switch (bw) {                                    \
        case 1: PDF_RES_SEM(1, F, __VA_ARGS__)       \
        case 2: PDF_RES_SEM(2, F, __VA_ARGS__)       \
        case 4: PDF_RES_SEM(4, F, __VA_ARGS__)       \
        case 8: PDF_RES_SEM(8, F, __VA_ARGS__)       \
        default: return cudaErrorInvalidValue;       \
    }

template <int BW, int SEM>
cudaError_t raise_batch_t(size_t smem) {
    return raise_smem_limit(reinterpret_cast<const void *>(k_batch_resident<BW, SEM>), smem);
}

}  // namespace

cudaError_t launch_resident(const FwdArgs &a, int sem, int out, uint32_t bw, uint32_t ctas, uint32_t threads,
                            size_t smem, cudaStream_t st) {
    PDF_RES(launch_t, a, out, ctas, threads, smem, st)
}
cudaError_t launch_fill_planes(const int8_t *value, uint32_t n_gates, uint64_t n_pairs, uint32_t *v, uint32_t *t,
                               uint32_t *m, uint64_t ld, uint32_t sms, cudaStream_t st) {
    const uint32_t W = (uint32_t)((n_pairs + 31) / 32), last = n_pairs & 31 ? (1u << (n_pairs & 31)) - 1u : 0xFFFFFFFFu;
    const uint32_t grid = std::min((n_gates + kFillThreads / 32 - 1) / (kFillThreads / 32), sms);
    const auto at16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (ld % 4 == 0 && at16(v) && at16(t) && at16(m)) k_fill_planes<true><<<grid, kFillThreads, 0, st>>>(value, n_gates, W, last, v, t, m, ld);
    else k_fill_planes<false><<<grid, kFillThreads, 0, st>>>(value, n_gates, W, last, v, t, m, ld);
    return cudaGetLastError();
}
cudaError_t prepare_resident_class(uint32_t sem, uint32_t bw, size_t smem) { PDF_RES(raise_batch_t, smem) }
cudaError_t launch_resident_class(const BatchLaunch &b, const BatchClass &c, cudaStream_t st) {
    const uint32_t sem = b.sem, bw = c.bw;
    PDF_RES(launch_batch_t, b, c, st)
}
