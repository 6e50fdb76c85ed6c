// pdf_wide.cu -- the wide forward kernel: the whole GPU on one level at a time.
//
// For circuits whose levels hold thousands of gates a walk per column block
// (forward_cta, forward_lanes_cta) is bound by instructions, about 200 per
// gate and 1,024 pairs, most of them for decoding the gate, its row addresses
// and its branches over again in every column block, and by having as many
// CTAs as column blocks: 32 of 148 SMs at 32,768 pairs.  Here the grid is one
// cooperative launch that takes the levels together, with a grid barrier
// after each: a warp takes one gate and a segment of up to 8 chunks of 32 LW
// words, decodes the gate once and runs its chunks in a tight loop, each lane
// LW consecutive words.  A row segment is up to 2 KB that one warp reads or
// writes whole.  What a level writes (2 rows of every gate) mostly stays in
// L2 for the level after it; rows are read past L1 (ld.global.cg), which is
// not coherent between SMs.
//
// Whether a gate holds a mark in a chunk is one bit of a byte per (segment,
// gate), written by the warp that owns the segment: no bitmap to clear and no
// atomics in the forward pass.
//
// Measured (B200, kernel, us): 150,000 gates without XOR, 40 levels, 32,768
// pairs, all planes stored, 4,032 (thread per gate) -> 1,200, of which the
// simulation alone is 545 (1.23 GB of rows written); 200,000 gates, 65,536 pairs, no
// planes: 1,733 -> 895.  What bounds it now is the end of each level, about 2 us
// of waiting for the last CTA and the grid's count, then the latency of a gate's
// record, mark flags and rows: 50,000 gates, 25 levels, 16,384 pairs, no planes
// (347 us): 23 warps of an issue wait at a barrier and 5 for memory, issue 22 %
// active, 115 MB of DRAM traffic, 4 % of its peak.
#include "pdf_kernels.cuh"
#include "pdf_ptx.cuh"

#include <cuda.h>

#include <algorithm>
#include <type_traits>

namespace {

template <int LW>
struct Words {
    uint32_t x[LW];
};
template <int LW>
__device__ __forceinline__ Words<LW> wload(const char *p) {  // past L1
    Words<LW> r;
    if constexpr (LW == 2) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2 *>(p));
        r.x[0] = v.x;
        r.x[1] = v.y;
    } else {
        r.x[0] = __ldcg(reinterpret_cast<const uint32_t *>(p));
    }
    return r;
}
template <int LW>
__device__ __forceinline__ Words<LW> wload_nc(const char *p) {  // inputs
    Words<LW> r;
    if constexpr (LW == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
        r.x[0] = v.x;
        r.x[1] = v.y;
    } else {
        r.x[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
    }
    return r;
}
// nw: the lane's words that hold pairs (the others are not written); once:
// nobody reads the row again
template <int LW>
__device__ __forceinline__ void wstore(char *p, const Words<LW> &v, uint32_t nw, bool once = false) {
    if constexpr (LW == 2) {
        if (nw == 2) {
            if (once) __stcs(reinterpret_cast<uint2 *>(p), make_uint2(v.x[0], v.x[1]));
            else *reinterpret_cast<uint2 *>(p) = make_uint2(v.x[0], v.x[1]);
        } else if (nw) {
            *reinterpret_cast<uint32_t *>(p) = v.x[0];
        }
    } else if (nw) {
        if (once) __stcs(reinterpret_cast<uint32_t *>(p), v.x[0]);
        else *reinterpret_cast<uint32_t *>(p) = v.x[0];
    }
}
template <int LW>
__device__ __forceinline__ Words<LW> wzero() {
    Words<LW> r;
#pragma unroll
    for (int j = 0; j < LW; j++) r.x[j] = 0;
    return r;
}
template <int LW>
__device__ __forceinline__ bool wany(const Words<LW> &v) {
    uint32_t o = 0;
#pragma unroll
    for (int j = 0; j < LW; j++) o |= v.x[j];
    return __any_sync(0xFFFFFFFFu, o != 0);
}

// One lane's place in a chunk: its first word, how many of its words hold
// pairs and their valid bits.
template <int LW>
struct Place {
    uint32_t w, nw;
    uint32_t wm[LW];
};
template <int LW>
__device__ __forceinline__ Place<LW> place(const FwdArgs &a, uint32_t chunk) {
    Place<LW> p;
    p.w = (chunk * 32 + (threadIdx.x & 31)) * LW;
    p.nw = p.w >= a.W ? 0u : min((uint32_t)LW, a.W - p.w);
#pragma unroll
    for (int j = 0; j < LW; j++)
        p.wm[j] = p.w + j + 1 < a.W ? 0xFFFFFFFFu
                                    : (p.w + j + 1 == a.W ? ((a.n_pairs & 31) ? (1u << (a.n_pairs & 31)) - 1u : 0xFFFFFFFFu)
                                                          : 0u);
    return p;
}

// The chunks [c0, c1) of gate g with NF = min(fan-ins, 4) fan-ins in the
// record (NF = 0: an input or a killed gate).  Returns the chunks that hold a
// mark, bit k for chunk c0 + k.
template <int SEM, int MODE, int LW, int NF>
__device__ __forceinline__ uint32_t wide_gate(const FwdArgs &a, const WideArgs &wa, uint32_t g, uint4 r0, uint4 r1,
                                              uint32_t seg, uint32_t c0, uint32_t c1) {
    constexpr bool FIX = SEM >= 2;
    const uint32_t h = r0.x, nfi = (h >> 8) & 0xFFu, nfold = hdr_nfold(h);
    const uint32_t ld4 = (uint32_t)(a.ld * 4), lb = (threadIdx.x & 31) * (LW * 4);
    const auto row = [&](const uint32_t *plane, uint32_t f) {
        return reinterpret_cast<const char *>(plane) + (size_t)f * ld4 + lb;
    };
    const uint32_t sw[4] = {r0.w, r1.x, r1.y, r1.z};
    const char *pv[NF ? NF : 1], *pt[NF ? NF : 1];
    uint32_t fz = 0;  // fan-ins that are the constant S0: their rows are not written (pdf_mark's given planes are)
#pragma unroll
    for (int q = 0; q < NF; q++) {
        const uint32_t f = sw[q] & ~SRC_ZERO;
        if (MODE != FWD_MARK && (sw[q] & SRC_ZERO)) fz |= 1u << q;
        pv[q] = row(a.V, f);
        pt[q] = row(a.T, f);
    }
    char *ov = const_cast<char *>(row(a.V, g)), *ot = const_cast<char *>(row(a.T, g)), *om = const_cast<char *>(row(a.M, g));
    const char *iv = nullptr, *it = nullptr;
    if (NF == 0 && (h & RF_INPT)) {
        const uint32_t pld4 = (uint32_t)(a.pi_ld * 4);
        iv = reinterpret_cast<const char *>(a.pi_v) + (size_t)r1.w * pld4 + lb;
        it = reinterpret_cast<const char *>(a.pi_t) + (size_t)r1.w * pld4 + lb;
    }
    // the chunks in which fan-in 0 (any fan-in in the FIXED modes) holds a mark
    uint32_t fm0 = 0, fmq[4] = {0, 0, 0, 0};
    const char *pm0 = nullptr;
    if (MODE != FWD_SIM && NF > 0) {
        const uint8_t *fl = wa.flags + (size_t)seg * a.c.n_gates;
        if (h & RF_MARKF0) {
            fm0 = __ldcg(fl + r1.w);
            pm0 = row(a.M, r1.w);
        }
        if (FIX && (h & RF_MANY))
#pragma unroll
            for (int q = 0; q < NF; q++) fmq[q] = __ldcg(fl + (sw[q] & ~SRC_ZERO));
    }
    const bool read_back = (h & RF_SPILL) != 0, keep_rows = a.store_all || read_back;
    // One chunk; returns whether the gate holds a mark in it.  FULL: every
    // word of the chunk holds 32 pairs; MK: a mark is possible.
    const auto chunk = [&](uint32_t c, auto full, auto may_mark) -> bool {
        constexpr bool FULL = decltype(full)::value, MK = MODE != FWD_SIM && decltype(may_mark)::value;
        const size_t o = (size_t)c * (128 * LW);
        const Place<LW> P = FULL ? Place<LW>{} : place<LW>(a, c);
        const bool live = FULL || P.nw != 0;
        const uint32_t nw = FULL ? (uint32_t)LW : P.nw;
        const bool m0 = MK && ((fm0 >> (c - c0)) & 1u);
        const auto far_row = [&](uint32_t q, Words<LW> &rv, Words<LW> &rt) {  // a fan-in past the fourth
            const uint32_t f = __ldg(a.c.edges + r0.z + q);
            rv = rt = wzero<LW>();
            if (live) {
                rv = wload<LW>(row(a.V, f) + o);
                rt = wload<LW>(row(a.T, f) + o);
            }
            return f;
        };
        Words<LW> V = wzero<LW>(), T = wzero<LW>(), M = wzero<LW>(), fv[NF ? NF : 1], ft[NF ? NF : 1];
        if (MODE == FWD_MARK) {  // the gate's own values are given
            if (live) {
                V = wload<LW>(ov + o);
                T = wload<LW>(ot + o);
            }
        } else if (NF == 0 && (h & RF_INPT)) {
            if (live) {
                V = wload_nc<LW>(iv + o);
                T = wload_nc<LW>(it + o);
            }
        } else if (NF == 0 && (h & RF_OINV)) {
#pragma unroll
            for (int j = 0; j < LW; j++) V.x[j] = 0xFFFFFFFFu;  // S0 inverted under both vectors: S1
        }
        // in the stage call pdf_mark fan-ins enter the side test only
        if (NF > 0 && (MODE != FWD_MARK || ((h & RF_SENS) && m0) || (FIX && (h & RF_MANY)))) {
#pragma unroll
            for (int q = 0; q < NF; q++) {
                fv[q] = ft[q] = wzero<LW>();
                if (live && !((fz >> q) & 1u)) {
                    fv[q] = wload<LW>(pv[q] + o);
                    ft[q] = wload<LW>(pt[q] + o);
                }
            }
        }
        if (m0 && live) M = wload<LW>(pm0 + o);
        if (NF > 0 && MODE != FWD_MARK) {
            uint32_t v1[LW];
#pragma unroll
            for (int j = 0; j < LW; j++) eval_first(h, fv[0].x[j], ft[0].x[j], V.x[j], v1[j]);
#pragma unroll
            for (int q = 1; q < NF; q++)
                if ((uint32_t)q <= nfold)
#pragma unroll
                    for (int j = 0; j < LW; j++) eval_fold<FIX>(h, V.x[j], v1[j], fv[q].x[j], ft[q].x[j]);
            if (NF == kInlineFanins)
                for (uint32_t q = kInlineFanins; q <= nfold; q++) {
                    Words<LW> rv, rt;
                    far_row(q, rv, rt);
#pragma unroll
                    for (int j = 0; j < LW; j++) eval_fold<FIX>(h, V.x[j], v1[j], rv.x[j], rt.x[j]);
                }
#pragma unroll
            for (int j = 0; j < LW; j++) eval_finish<FIX>(h, V.x[j], v1[j], T.x[j]);
        }
        if constexpr (!FULL) {
#pragma unroll
            for (int j = 0; j < LW; j++) {
                V.x[j] &= P.wm[j];
                T.x[j] &= P.wm[j];
            }
        }
        bool marked = false;
        if constexpr (MK) {  // markkernel.cuh:226-267
            if (NF == 0) {
                if ((h & RF_INPT) && (h & RF_MARKF0)) {
                    M = T;
                    marked = wany<LW>(M);
                }
            } else if (m0) {
#pragma unroll
                for (int j = 0; j < LW; j++) M.x[j] &= T.x[j];
                marked = wany<LW>(M);
                if ((h & RF_SENS) && marked) {
                    SensAcc s[LW];
                    const bool or_like = (h & RF_IM) != 0;
#pragma unroll
                    for (int j = 0; j < LW; j++) sens_init(s[j]);
#pragma unroll
                    for (int q = 0; q < NF; q++)
#pragma unroll
                        for (int j = 0; j < LW; j++) sens_step<SEM & 1>(s[j], or_like, fv[q].x[j], ft[q].x[j]);
                    if (NF == kInlineFanins)
                        for (uint32_t q = kInlineFanins; q < nfi; q++) {
                            Words<LW> rv, rt;
                            far_row(q, rv, rt);
#pragma unroll
                            for (int j = 0; j < LW; j++) sens_step<SEM & 1>(s[j], or_like, rv.x[j], rt.x[j]);
                        }
#pragma unroll
                    for (int j = 0; j < LW; j++) M.x[j] &= sens_result<SEM & 1>(s[j]);
                    marked = wany<LW>(M);
                }
            } else if (FIX && (h & RF_MANY) && wany<LW>(T)) {
                const uint32_t mor = flagmask(h, RF_IM), mxor = flagmask(h, RF_XOR), mand = ~(mor | mxor);
                SensAcc s[LW];
#pragma unroll
                for (int j = 0; j < LW; j++) sens_init(s[j]);
                const auto step = [&](const Words<LW> &rv, const Words<LW> &rt, uint32_t f, bool holds) {
                    Words<LW> rm = wzero<LW>();
                    if (live && holds) rm = wload<LW>(row(a.M, f) + o);
#pragma unroll
                    for (int j = 0; j < LW; j++)
                        sens_step_fixed<SEM == PDF_MARK_FIXED_NONROBUST>(s[j], mand, mor, mxor, rv.x[j], rt.x[j], rm.x[j]);
                };
#pragma unroll
                for (int q = 0; q < NF; q++) step(fv[q], ft[q], sw[q] & ~SRC_ZERO, (fmq[q] >> (c - c0)) & 1u);
                if (NF == kInlineFanins)
                    for (uint32_t q = kInlineFanins; q < nfi; q++) {
                        Words<LW> rv, rt;
                        const uint32_t f = far_row(q, rv, rt);
                        step(rv, rt, f, (__ldcg(wa.flags + (size_t)seg * a.c.n_gates + f) >> (c - c0)) & 1u);
                    }
#pragma unroll
                for (int j = 0; j < LW; j++) M.x[j] = T.x[j] & sens_result<SEM == PDF_MARK_FIXED_NONROBUST>(s[j]);
                marked = wany<LW>(M);
            }
        }
        // rows that no gate reads again leave L2 to the others (streaming stores)
        if (MODE != FWD_MARK && (keep_rows || marked)) {
            wstore<LW>(ov + o, V, nw, !read_back);
            wstore<LW>(ot + o, T, nw, !read_back);
        }
        if (MODE != FWD_SIM && (a.store_all || marked)) {
            if constexpr (!MK) M = wzero<LW>();
            wstore<LW>(om + o, M, nw, !marked);
        }
        return marked;
    };
    uint32_t marks = 0;
    const uint32_t cf = max(c0, min(c1, (uint32_t)(a.n_pairs / (1024 * LW))));  // full chunks end here
    const bool may = NF == 0 ? (h & RF_INPT) && (h & RF_MARKF0) : fm0 || (FIX && (h & RF_MANY));
    if (!may) {
        uint32_t c = c0;
        if constexpr (NF > 0 && MODE != FWD_MARK) {
            // no mark to form: the rows of several chunks in flight
            constexpr int U = 2;
            if (nfi <= kInlineFanins)
                for (; c + U <= cf; c += U) {
                    Words<LW> fv[U][NF], ft[U][NF];
#pragma unroll
                    for (int u = 0; u < U; u++)
#pragma unroll
                        for (int q = 0; q < NF; q++) {
                            fv[u][q] = ft[u][q] = wzero<LW>();
                            if (!((fz >> q) & 1u)) {
                                fv[u][q] = wload<LW>(pv[q] + (size_t)(c + u) * (128 * LW));
                                ft[u][q] = wload<LW>(pt[q] + (size_t)(c + u) * (128 * LW));
                            }
                        }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const size_t o = (size_t)(c + u) * (128 * LW);
                        Words<LW> V, T;
                        uint32_t v1[LW];
#pragma unroll
                        for (int j = 0; j < LW; j++) eval_first(h, fv[u][0].x[j], ft[u][0].x[j], V.x[j], v1[j]);
#pragma unroll
                        for (int q = 1; q < NF; q++)
                            if ((uint32_t)q <= nfold)
#pragma unroll
                                for (int j = 0; j < LW; j++)
                                    eval_fold<FIX>(h, V.x[j], v1[j], fv[u][q].x[j], ft[u][q].x[j]);
#pragma unroll
                        for (int j = 0; j < LW; j++) eval_finish<FIX>(h, V.x[j], v1[j], T.x[j]);
                        if (keep_rows) {
                            wstore<LW>(ov + o, V, LW, !read_back);
                            wstore<LW>(ot + o, T, LW, !read_back);
                        }
                        if (MODE != FWD_SIM && a.store_all) wstore<LW>(om + o, wzero<LW>(), LW, true);
                    }
                }
        }
        for (; c < cf; c++) (void)chunk(c, std::true_type{}, std::false_type{});
    } else {
        for (uint32_t c = c0; c < cf; c++)
            if (chunk(c, std::true_type{}, std::true_type{})) marks |= 1u << (c - c0);
    }
    for (uint32_t c = cf; c < c1; c++)
        if (chunk(c, std::false_type{}, std::true_type{})) marks |= 1u << (c - c0);
    return marks;
}

// All CTAs of the (cooperative) grid; what each wrote before is visible after.
// Bounded: false when the others did not come within `polls` (0: 2^22, seconds).
__device__ __forceinline__ uint32_t acquire_u32(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool grid_sync(WideSync *s, uint32_t target, uint32_t polls) {
    __threadfence();
    atomicAdd(&s->arrived, 1u);
    if (polls) {
        for (uint32_t i = 0; i < polls; i++)
            if (acquire_u32(&s->arrived) >= target) return true;
        return false;
    }
    for (uint32_t i = 0; i < (1u << 22); i++)
        if (acquire_u32(&s->arrived) >= target) return true;
    return false;
}

template <int SEM, int MODE, int LW>
__global__ void __launch_bounds__(kWideThreads, kWideCtas) k_wide(const FwdArgs a, const WideArgs wa) {
    __shared__ uint32_t s_reach, s_top, s_seen, s_fail, s_next;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t gt = blockIdx.x * blockDim.x + tid, GT = gridDim.x * blockDim.x;
    const uint32_t G = a.c.n_gates, L = a.c.n_levels;
    const uint32_t nf = (a.W + kLaneCoverWords - 1) / kLaneCoverWords;  // cover bitmaps
    uint32_t phase = 0, told = 0;
    if (tid == 0) {
        s_reach = 0;
        s_top = 0;
        s_fail = 0;
        s_next = 0;
    }
    if (MODE == FWD_FUSED) {  // the batch's cover state (the cover kernels run after this one)
        for (size_t i = gt; i < (size_t)nf * a.bm_words; i += GT) a.nzb_fine[i] = 0;
        // no marked level, should this CTA leave before the prune
        for (uint32_t b = gt; b < nf; b += GT) a.maxlvl_fine[b] = 0;
        if (a.active)
            for (uint32_t w = gt; w <= a.W; w += GT) a.active[w] = 0;
        if (a.acc && gt == 0) {
            a.acc->batch_lo = 0;
            a.acc->batch_hi = 0;
            a.acc->batch_flags = 0;
            a.acc->done = 0;
            a.acc->n_over = 0;
            a.acc->done_over = 0;
        }
    }
    __syncthreads();
    // The CTA's items of a level are every gridDim-th; its warps take them as
    // they come free (a gate that holds marks costs several times one that
    // does not).
    const auto next_item = [&]() -> uint32_t {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&s_next, 1u);
        return __shfl_sync(0xFFFFFFFFu, k, 0) * gridDim.x + blockIdx.x;
    };
    // After a level: this CTA's findings out, everyone's in.  Returns false
    // when the grid did not come together.
    const auto level_done = [&]() -> bool {
        __syncthreads();
        if (tid == 0) {
            if (MODE != FWD_SIM && s_top != told) {
                told = s_top;
                atomicMax(&wa.sync->reach, s_reach);
                atomicMax(&wa.sync->top, s_top);
            }
            if (!grid_sync(wa.sync, ++phase * gridDim.x, a.wait_polls)) s_fail = 1;
            s_seen = MODE != FWD_SIM ? __ldcg(&wa.sync->reach) : 0u;
            s_next = 0;
        }
        __syncthreads();
        return s_fail == 0;
    };
    const auto finish = [&](bool ok) {  // the last CTA leaves the counters as it found them
        __syncthreads();
        if (tid != 0) return;
        if (!ok) atomicOr(a.err, kErrTimeout);
        __threadfence();
        if (atomicAdd(&wa.sync->left, 1u) == gridDim.x - 1) {
            wa.sync->arrived = 0;
            wa.sync->left = 0;
            wa.sync->reach = 0;
            wa.sync->top = 0;
        }
    };
    // ------------------------------------------------------------- forward
    const bool early = MODE != FWD_SIM && a.in_pieces;
    const uint32_t cps = wa.cps, nseg = wa.nseg;
    bool ok = true;
    for (uint32_t l = 0; l < L && ok; l++) {
        const uint32_t ga = __ldg(a.c.level_off + l), n = __ldg(a.c.level_off + l + 1) - ga;
        uint32_t reach = 0;
        bool any = false;
        // the next item's gate and record, loaded an item ahead
        uint32_t i1 = 0, seg1 = 0, g1 = 0;
        uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
        const auto fetch = [&]() {
            i1 = next_item();
            if (i1 >= n * nseg) return;
            seg1 = nseg == 1 ? 0u : i1 / n;
            g1 = ga + i1 - seg1 * n;
            const uint4 *rp = reinterpret_cast<const uint4 *>(a.c.rec + g1);
            n0 = __ldg(rp);
            n1 = __ldg(rp + 1);
        };
        fetch();
        while (i1 < n * nseg) {
            const uint32_t seg = seg1, g = g1;
            const uint32_t c0 = seg * cps, c1 = min(wa.chunks, c0 + cps);
            const uint4 r0 = n0, r1 = n1;
            fetch();
            // a killed gate needs no fan-in, but for pdf_mark's given values
            const uint32_t nfi =
                (r0.x & (MODE == FWD_MARK ? RF_INPT : RF_INPT | RF_KILL)) ? 0u : (r0.x >> 8) & 0xFFu;
            uint32_t m;
            switch (min(nfi, 4u)) {
                case 0: m = wide_gate<SEM, MODE, LW, 0>(a, wa, g, r0, r1, seg, c0, c1); break;
                case 1: m = wide_gate<SEM, MODE, LW, 1>(a, wa, g, r0, r1, seg, c0, c1); break;
                case 2: m = wide_gate<SEM, MODE, LW, 2>(a, wa, g, r0, r1, seg, c0, c1); break;
                case 3: m = wide_gate<SEM, MODE, LW, 3>(a, wa, g, r0, r1, seg, c0, c1); break;
                default: m = wide_gate<SEM, MODE, LW, 4>(a, wa, g, r0, r1, seg, c0, c1); break;
            }
            if (MODE != FWD_SIM) {
                if (lane == 0) wa.flags[(size_t)seg * G + g] = (uint8_t)m;
                if (m) {
                    any = true;
                    reach = max(reach, r0.y >> 16);
                }
            }
        }
        if (MODE != FWD_SIM && any && lane == 0) {
            s_top = l + 1;  // the same from every warp
            if (reach > l) atomicMax(&s_reach, reach);
        }
        if (l + 1 == L && MODE == FWD_SIM) break;
        ok = level_done();
        if (early && s_seen <= l) {  // no gate above can be marked
            if (MODE == FWD_MARK) {   // the rows left out hold no mark
                for (uint32_t g = ga + n + blockIdx.x; g < G; g += gridDim.x)
                    for (uint32_t x = tid; x < a.W; x += blockDim.x) __stcs(a.M + (size_t)g * a.ld + x, 0u);
            }
            break;
        }
    }
    if (MODE == FWD_SIM || !ok || (MODE == FWD_MARK && a.no_prune)) {
        finish(ok);
        return;
    }
    // ------------------------------------------------------ prune and merge
    // levels descending; a gate's pruned mark is final once its fan-outs' are.
    // Gates from level `top` on hold no mark (past the last level walked their
    // flags are not this launch's).
    if (tid == 0) s_top = __ldcg(&wa.sync->top);
    __syncthreads();
    const uint32_t top = s_top, g_top = __ldg(a.c.level_off + top);
    if (MODE == FWD_FUSED)
        for (uint32_t b = gt; b < nf; b += GT) a.maxlvl_fine[b] = top;
    const uint32_t ld4 = (uint32_t)(a.ld * 4), lb = lane * (LW * 4);
    constexpr uint32_t kSub = kLaneCoverWords / LW;  // lanes per cover bitmap
    constexpr uint32_t kPer = 32 / kSub;             // cover bitmaps per chunk
    constexpr int kB = 4;                            // chunks in flight
    for (int l = (int)top - 1; l >= 0 && ok; l--) {
        const uint32_t ga = __ldg(a.c.level_off + l), n = __ldg(a.c.level_off + l + 1) - ga, items = n * nseg;
        const auto flag_of = [&](uint32_t i, uint32_t &seg, uint32_t &g) -> uint32_t {
            seg = nseg == 1 ? 0u : i / n;
            g = ga + i - seg * n;
            return __ldcg(wa.flags + (size_t)seg * G + g);
        };
        uint32_t i1 = next_item(), seg1 = 0, g1 = 0, m1 = i1 < items ? flag_of(i1, seg1, g1) : 0u;  // the next item's
        while (i1 < items) {
            const uint32_t seg = seg1, g = g1, m = m1;
            i1 = next_item();
            if (i1 < items) m1 = flag_of(i1, seg1, g1);
            if (!m) continue;
            uint8_t *fl = wa.flags + (size_t)seg * G;
            const uint4 r0 = __ldg(reinterpret_cast<const uint4 *>(a.c.rec + g));
            const bool po = (r0.x >> 4) & 1u;
            const uint32_t nfo = po ? 0u : r0.y & a.c.nfo_mask, base = r0.z + ((r0.x >> 8) & 0xFFu);
            // 32 fan-outs at a time, one per lane: id and the chunks it is marked in
            const auto fanouts = [&](uint32_t k0, uint32_t &fo, uint32_t &fb) {
                fo = k0 + lane < nfo ? __ldg(a.c.edges + base + k0 + lane) : kEmpty;
                fb = fo < g_top ? __ldcg(fl + fo) & m : 0u;
            };
            uint32_t fo0, fb0;
            fanouts(0, fo0, fb0);
            char *mrow = reinterpret_cast<char *>(a.M) + (size_t)g * ld4 + lb;
            uint32_t left = 0, px = kEmpty, py = kEmpty;
            for (uint32_t b0 = 0; b0 < cps; b0 += kB) {
                const uint32_t mm = (m >> b0) & ((1u << kB) - 1u);
                if (!mm) continue;
                const uint32_t c = seg * cps + b0;
                // words of the lane that hold pairs, over the chunks (rows hold no
                // bit past the last pair)
                const uint32_t w0 = (c * 32 + lane) * LW;
                const auto words = [&](int u) -> uint32_t {
                    const uint32_t w = w0 + u * 32 * LW;
                    return w >= a.W ? 0u : min((uint32_t)LW, a.W - w);
                };
                Words<LW> mk[kB], keep[kB];
#pragma unroll
                for (int u = 0; u < kB; u++) {
                    mk[u] = wzero<LW>();
                    if (((mm >> u) & 1u) && words(u)) {
                        mk[u] = wload<LW>(mrow + (size_t)(c + u) * (128 * LW));
                        // (a lane's second word may lie past the last pair)
                        if (LW == 2 && words(u) == 1) mk[u].x[LW - 1] = 0;
                    }
#pragma unroll
                    for (int j = 0; j < LW; j++) keep[u].x[j] = po ? 0xFFFFFFFFu : 0u;
                }
                for (uint32_t k0 = 0; k0 < nfo; k0 += 32) {
                    uint32_t fo = fo0, fb = fb0;
                    if (k0) fanouts(k0, fo, fb);
                    uint32_t todo = __ballot_sync(0xFFFFFFFFu, (fb >> b0) & mm);
                    while (todo) {  // a marked fan-out's chunks together
                        const int k = __ffs(todo) - 1;
                        todo &= todo - 1;
                        const uint32_t f = __shfl_sync(0xFFFFFFFFu, fo, k);
                        const uint32_t fm = (__shfl_sync(0xFFFFFFFFu, fb, k) >> b0) & mm;
                        const char *frow = reinterpret_cast<const char *>(a.M) + (size_t)f * ld4 + lb;
                        Words<LW> q[kB];
#pragma unroll
                        for (int u = 0; u < kB; u++) {
                            q[u] = wzero<LW>();
                            if (((fm >> u) & 1u) && words(u)) q[u] = wload<LW>(frow + (size_t)(c + u) * (128 * LW));
                        }
#pragma unroll
                        for (int u = 0; u < kB; u++)
#pragma unroll
                            for (int j = 0; j < LW; j++) keep[u].x[j] |= q[u].x[j];
                    }
                }
                uint32_t zs = 0;  // the chunks that keep a mark
#pragma unroll
                for (int u = 0; u < kB; u++) {
                    bool changed = false;
                    uint32_t some = 0;
#pragma unroll
                    for (int j = 0; j < LW; j++) {
                        const uint32_t nm = mk[u].x[j] & keep[u].x[j];
                        changed |= nm != mk[u].x[j];
                        some |= nm;
                        mk[u].x[j] = nm;
                    }
                    if (changed) wstore<LW>(mrow + (size_t)(c + u) * (128 * LW), mk[u], words(u));
                    const uint32_t z = __ballot_sync(0xFFFFFFFFu, some != 0);
                    if (!z) continue;
                    zs |= 1u << u;
                    // the cover's bitmap of every 8 words that keep a mark
                    if (MODE == FWD_FUSED && lane < kPer && ((z >> (kSub * lane)) & ((1u << kSub) - 1u)))
                        atomicOr(a.nzb_fine + (size_t)((c + u) * kPer + lane) * a.bm_words + (g >> 5), 1u << (g & 31));
                }
                left |= zs << b0;
                if (MODE == FWD_FUSED && a.first_x && zs) {  // first falling / rising pair of each lane
                    Words<LW> v[kB];
#pragma unroll
                    for (int u = 0; u < kB; u++) {
                        v[u] = wzero<LW>();
                        if (((zs >> u) & 1u) && words(u))
                            v[u] = wload<LW>(reinterpret_cast<const char *>(a.V) + (size_t)g * ld4 + lb +
                                             (size_t)(c + u) * (128 * LW));
                    }
#pragma unroll
                    for (int u = 0; u < kB; u++)
#pragma unroll
                        for (int j = 0; j < LW; j++) {
                            const uint32_t fx = mk[u].x[j] & ~v[u].x[j], fy = mk[u].x[j] & v[u].x[j];
                            if (fx) px = min(px, (w0 + u * 32 * LW + j) * 32 + (__ffs(fx) - 1));
                            if (fy) py = min(py, (w0 + u * 32 * LW + j) * 32 + (__ffs(fy) - 1));
                        }
                }
            }
            if (left != m && lane == 0) fl[g] = (uint8_t)left;
            if (MODE == FWD_FUSED && a.first_x && left) {
                px = __reduce_min_sync(0xFFFFFFFFu, px);
                py = __reduce_min_sync(0xFFFFFFFFu, py);
                if (lane == 0) {
                    const uint32_t id = net_id(a.c, g);
                    if (px != kEmpty) atomicMin(a.first_x + id, a.pair_base + px);
                    if (py != kEmpty) atomicMin(a.first_y + id, a.pair_base + py);
                }
            }
        }
        if (l) ok = level_done();
    }
    finish(ok);
}

template <int SEM, int MODE, int LW>
cudaError_t launch_t(const FwdArgs &a, const WideArgs &wa, uint32_t sms, cudaStream_t st) {
    FwdArgs fa = a;
    WideArgs w = wa;
    void *args[] = {&fa, &w};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_wide<SEM, MODE, LW>), dim3(sms * kWideCtas),
                                       dim3(kWideThreads), args, 0, st);
}
template <int SEM, int LW>
cudaError_t launch_mode(const FwdArgs &a, const WideArgs &wa, int mode, uint32_t sms, cudaStream_t st) {
    switch (mode) {
        case FWD_FUSED: return launch_t<SEM, FWD_FUSED, LW>(a, wa, sms, st);
        case FWD_SIM: return launch_t<SEM, FWD_SIM, LW>(a, wa, sms, st);
        default: return launch_t<SEM, FWD_MARK, LW>(a, wa, sms, st);
    }
}
template <int LW>
cudaError_t launch_sem(const FwdArgs &a, const WideArgs &wa, int mode, int sem, uint32_t sms, cudaStream_t st) {
    switch (sem) {
        case 0: return launch_mode<0, LW>(a, wa, mode, sms, st);
        case 1: return launch_mode<1, LW>(a, wa, mode, sms, st);
        case 2: return launch_mode<2, LW>(a, wa, mode, sms, st);
        case 3: return launch_mode<3, LW>(a, wa, mode, sms, st);
        default: return cudaErrorInvalidValue;
    }
}

// SMs that a kernel on `st` can take, at most `sms`: a stream of a green context
// has a part of the device's, and a cooperative grid has to fit it.
uint32_t stream_sms(cudaStream_t st, uint32_t sms) {
    using GetCtx = CUresult (*)(CUstream, CUcontext *, CUgreenCtx *);
    using GetRes = CUresult (*)(CUgreenCtx, CUdevResource *, CUdevResourceType);
    static const auto entry = [](const char *name) -> void * {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion(name, &f, 12050, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return f;
        (void)cudaGetLastError();
        return nullptr;
    };
    static const GetCtx get_ctx = reinterpret_cast<GetCtx>(entry("cuStreamGetCtx"));
    static const GetRes get_res = reinterpret_cast<GetRes>(entry("cuGreenCtxGetDevResource"));
    CUcontext ctx = nullptr;
    CUgreenCtx green = nullptr;
    CUdevResource res{};
    if (!get_ctx || !get_res || get_ctx(st, &ctx, &green) != CUDA_SUCCESS || !green ||
        get_res(green, &res, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS || !res.sm.smCount)
        return sms;
    return std::min(sms, res.sm.smCount);
}

}  // namespace

cudaError_t launch_wide(const FwdArgs &a, const WideArgs &wa, int mode, int sem, uint32_t lw, uint32_t sms,
                        cudaStream_t st) {
    if (!wa.chunks || !wa.cps || wa.cps > 8) return cudaErrorInvalidValue;
    sms = stream_sms(st, sms);
    return lw == 2 ? launch_sem<2>(a, wa, mode, sem, sms, st) : launch_sem<1>(a, wa, mode, sem, sms, st);
}
