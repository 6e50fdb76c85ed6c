// pdf_lanes.cu -- the lane forward kernel: a warp per gate.
#include "pdf_kernels.cuh"
#include "pdf_ptx.cuh"

#include <algorithm>

namespace {

// ---------------------------------------------------------------------------
// Lane forward kernel (tiles of 32 x LW words, LW = 1 or 2): the same stages
// as forward_cta (sim, forward mark, prune, merge) with the roles of threads
// turned around.  Lane j of every warp carries words w0 + LW j .. + LW - 1 of
// the column block, and a warp evaluates one gate at a time for the whole
// block, so every instruction of a gate is uniform across the warp (no
// divergence on gate type or fan-in count), a gate's record is decoded once
// per 1,024 LW pairs, and every plane-row access is one coalesced line of
// 128 LW bytes.  Warps take the gates of a level in turn; the gates of a
// level depend only on lower levels, so a CTA needs one barrier per level
// (not per piece of a level), and every fan-in is read from its plane row
// (L1/L2), which is what wide levels need: nothing of the circuit is kept on
// chip except the block's mark bitmap and the staged records.  Several gates
// per warp are in flight at a time (their fan-in rows are loaded before any
// is evaluated).
//
// Every gate with fan-outs writes its V and T rows (its readers load them);
// a gate writes its M row only when it holds a mark (every reader of a mark
// row tests the gate's bitmap bit first), or when the caller asked for the
// planes (store_all).  Words past the last pair of a row are read (rows are
// padded to whole blocks) but masked, and never written.
// ---------------------------------------------------------------------------

// A lane's view of the planes: its first word in row 0 of each plane, and
// the row pitch in bytes (below 2^32: planes_fit), so that a row address is
// one wide multiply-add.
struct LanePlanes {
    char *V, *T, *M;
    uint32_t ld4;
};
template <typename P>
__device__ __forceinline__ uint32_t *lrow(P *base, uint32_t f, uint32_t ld4) {
    return reinterpret_cast<uint32_t *>(const_cast<char *>(base) + (size_t)f * ld4);
}
template <int LW>
__device__ __forceinline__ void lload(const uint32_t *p, uint32_t (&d)[LW]) {
    if constexpr (LW == 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(p);
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
        d[3] = v.w;
    } else if constexpr (LW == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        d[0] = v.x;
        d[1] = v.y;
    } else {
        d[0] = *p;
    }
}
template <int LW>
__device__ __forceinline__ void lload_nc(const uint32_t *p, uint32_t (&d)[LW]) {
    if constexpr (LW == 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
        d[3] = v.w;
    } else if constexpr (LW == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
        d[0] = v.x;
        d[1] = v.y;
    } else {
        d[0] = __ldg(p);
    }
}
// nw: the lane's words that hold pairs (1..LW); the others are not written
template <int LW>
__device__ __forceinline__ void lstore(uint32_t *p, const uint32_t (&s)[LW], uint32_t nw) {
    if constexpr (LW == 4) {
        if (nw == 4) {
            *reinterpret_cast<uint4 *>(p) = make_uint4(s[0], s[1], s[2], s[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 3; j++)
                if ((uint32_t)j < nw) p[j] = s[j];
        }
    } else if constexpr (LW == 2) {
        if (nw == 2) *reinterpret_cast<uint2 *>(p) = make_uint2(s[0], s[1]);
        else p[0] = s[0];
    } else {
        p[0] = s[0];
    }
}
template <int LW>
__device__ __forceinline__ void lzero(uint32_t (&d)[LW]) {
#pragma unroll
    for (int j = 0; j < LW; j++) d[j] = 0;
}
template <int LW>
__device__ __forceinline__ bool lany(const uint32_t (&d)[LW]) {
    uint32_t o = 0;
#pragma unroll
    for (int j = 0; j < LW; j++) o |= d[j];
    return o != 0;
}

// Fan-in rows of one gate, loaded before it is evaluated (its record stays
// in shared memory; the header travels here).
template <int LW>
struct LaneIn {
    uint32_t h;                          // record header
    uint32_t fv[kInlineFanins][LW], ft[kInlineFanins][LW];
    uint32_t m0[LW];                     // mark row of fan-in 0 (when its bitmap bit is set)
    uint32_t fm[kInlineFanins][LW];      // FIXED modes: mark rows of fan-ins 0..3 with their bits set
    uint32_t sv[LW], st[LW];             // stage call pdf_mark: the gate's own given V and T
    bool bit0;                           // fan-in 0 holds a mark in this column block
};

template <int SEM, int MODE, int LW>
__device__ __forceinline__ void lane_load(const FwdArgs &a, const LanePlanes &P, const uint32_t *bm,
                                          const GateRec *rp, uint32_t g, uint32_t w, bool live, LaneIn<LW> &x) {
    constexpr bool FIX = SEM >= 2;
    const uint4 r0 = reinterpret_cast<const uint4 *>(rp)[0], r1 = reinterpret_cast<const uint4 *>(rp)[1];
    const uint32_t h = r0.x, nfi = (h >> 8) & 0xFFu;
    x.h = h;
    // Whether fan-in 0 holds a mark in the block: the same on every lane of
    // the warp (the branch in lane_gate that it guards holds warp votes), so
    // it is set before any lane leaves.  m0 is read only where bit0 and
    // RF_MARKF0 had it loaded.
    x.bit0 = MODE != FWD_SIM && !(h & (RF_INPT | RF_KILL)) && bit_test(bm, r1.w);
    // A lane past the last pair loads nothing: what it evaluates is masked.
    if (!live) return;
    if (h & RF_INPT) {
        if (MODE == FWD_MARK) {
            lload<LW>(lrow(P.V, g, P.ld4), x.fv[0]);
            lload<LW>(lrow(P.T, g, P.ld4), x.ft[0]);
        } else {
            const uint32_t pld4 = (uint32_t)(a.pi_ld * 4);
            lload_nc<LW>(lrow(reinterpret_cast<const char *>(a.pi_v + w), r1.w, pld4), x.fv[0]);
            lload_nc<LW>(lrow(reinterpret_cast<const char *>(a.pi_t + w), r1.w, pld4), x.ft[0]);
        }
        return;
    }
    if (MODE == FWD_MARK) {  // the gate's own values are given; fan-ins feed the side test only
        lload<LW>(lrow(P.V, g, P.ld4), x.sv);
        lload<LW>(lrow(P.T, g, P.ld4), x.st);
    }
    // A killed gate's value is S0 whatever its fan-ins (and it cannot mark):
    // nothing to load.  Fan-ins 0 .. nl - 1 follow warp-uniform branches on
    // the count, so absent fan-ins cost no predicated-off slots; a killed
    // fan-in is S0 (its row is not written), except in the stage call
    // pdf_mark, whose given planes are read as they are.
    if (h & RF_KILL) return;
    const uint32_t nl = min(nfi, (uint32_t)kInlineFanins);
    const auto fanin = [&](int q, uint32_t sw) {
        const uint32_t f = sw & ~SRC_ZERO;
        if (MODE == FWD_MARK || !(sw & SRC_ZERO)) {
            lload<LW>(lrow(P.V, f, P.ld4), x.fv[q]);
            lload<LW>(lrow(P.T, f, P.ld4), x.ft[q]);
        } else {
            lzero<LW>(x.fv[q]);
            lzero<LW>(x.ft[q]);
        }
        if (FIX && MODE != FWD_SIM) {
            if (bit_test(bm, f)) lload<LW>(lrow(P.M, f, P.ld4), x.fm[q]);
            else lzero<LW>(x.fm[q]);
        }
    };
    if (nl > 0) {
        fanin(0, r0.w);
        if (nl > 1) {
            fanin(1, r1.x);
            if (nl > 2) {
                fanin(2, r1.y);
                if (nl > 3) fanin(3, r1.z);
            }
        }
    }
    if (MODE != FWD_SIM && (h & RF_MARKF0) && x.bit0) lload<LW>(lrow(P.M, r1.w, P.ld4), x.m0);
}

// Evaluate, mark and store one gate; returns whether it holds a mark in the
// block (warp-uniform).  wm: the lane's word masks (pairs present); reach (in
// shared memory) grows to the last level that a marked gate carries to: kept by
// the caller in registers it spilled the forward pass (64-word tile, 183,874
// gates, planes: 6.6 -> 7.7 ms).
template <int SEM, int MODE, int LW>
__device__ __forceinline__ bool lane_gate(const FwdArgs &a, const LanePlanes &P, uint32_t *bm, const GateRec *rp,
                                          uint32_t g, bool live, uint32_t nw, const uint32_t (&wm)[LW],
                                          uint32_t *reach, const LaneIn<LW> &x) {
    constexpr bool FIX = SEM >= 2;
    const uint32_t h = x.h, nfi = (h >> 8) & 0xFFu;
    // fan-in q > 3 of the gate (its id from the edge array), read from its rows
    const auto far_row = [&](uint32_t q, uint32_t (&v)[LW], uint32_t (&t)[LW]) {
        const uint32_t f = __ldg(a.c.edges + rp->w[2] + q);
        lzero<LW>(v);
        lzero<LW>(t);
        if (live) {
            lload<LW>(lrow(P.V, f, P.ld4), v);
            lload<LW>(lrow(P.T, f, P.ld4), t);
        }
        return f;
    };
    uint32_t V[LW], T[LW], M[LW];
    lzero<LW>(M);
    if (h & RF_INPT) {
#pragma unroll
        for (int j = 0; j < LW; j++) {
            V[j] = x.fv[0][j] & wm[j];
            T[j] = x.ft[0][j] & wm[j];
        }
    } else if (MODE == FWD_MARK) {
#pragma unroll
        for (int j = 0; j < LW; j++) {
            V[j] = x.sv[j] & wm[j];
            T[j] = x.st[j] & wm[j];
        }
    } else if ((h & RF_KILL) || !live) {
        lzero<LW>(V);
        lzero<LW>(T);
        if (h & RF_OINV) {
#pragma unroll
            for (int j = 0; j < LW; j++) V[j] = wm[j];  // S0 inverted under both vectors: S1
        }
    } else {
        uint32_t v1[LW];
#pragma unroll
        for (int j = 0; j < LW; j++) eval_first(h, x.fv[0][j], x.ft[0][j], V[j], v1[j]);
        // fold steps in fan-in order, behind warp-uniform branches on the count
        const uint32_t nfold = hdr_nfold(h);
        const auto fold = [&](int q) {
#pragma unroll
            for (int j = 0; j < LW; j++) eval_fold<FIX>(h, V[j], v1[j], x.fv[q][j], x.ft[q][j]);
        };
        if (nfold >= 1) {
            fold(1);
            if (nfold >= 2) {
                fold(2);
                if (nfold >= 3) fold(3);
            }
        }
        for (uint32_t q = kInlineFanins; q <= nfold; q++) {
            uint32_t rv[LW], rt[LW];
            far_row(q, rv, rt);
#pragma unroll
            for (int j = 0; j < LW; j++) eval_fold<FIX>(h, V[j], v1[j], rv[j], rt[j]);
        }
#pragma unroll
        for (int j = 0; j < LW; j++) {
            eval_finish<FIX>(h, V[j], v1[j], T[j]);
            V[j] &= wm[j];
            T[j] &= wm[j];
        }
    }
    if (MODE != FWD_SIM) {  // markkernel.cuh:226-267
        const bool anyT = __any_sync(0xFFFFFFFFu, lany<LW>(T));
        if (h & RF_INPT) {
            // (the whole netlist's inputs always)
            const uint32_t on = MODE == FWD_MARK ? 0xFFFFFFFFu : flagmask(h, RF_MARKF0);
#pragma unroll
            for (int j = 0; j < LW; j++) M[j] = T[j] & on;
        } else if ((h & RF_MARKF0) && x.bit0 && anyT) {
            // fan-in 0 (gate w[7]) holds a mark: its bitmap bit is set
#pragma unroll
            for (int j = 0; j < LW; j++) M[j] = T[j] & x.m0[j];
            if ((h & RF_SENS) && __any_sync(0xFFFFFFFFu, lany<LW>(M))) {
                // the side test over the fan-in rows already loaded (past the
                // fourth, read here)
                SensAcc s[LW];
                const bool or_like = (h & RF_IM) != 0;
#pragma unroll
                for (int j = 0; j < LW; j++) sens_init(s[j]);
#pragma unroll
                for (int q = 0; q < kInlineFanins; q++)
                    if ((uint32_t)q < nfi)
#pragma unroll
                        for (int j = 0; j < LW; j++) sens_step<SEM & 1>(s[j], or_like, x.fv[q][j], x.ft[q][j]);
                for (uint32_t q = kInlineFanins; q < nfi; q++) {
                    uint32_t rv[LW], rt[LW];
                    far_row(q, rv, rt);
#pragma unroll
                    for (int j = 0; j < LW; j++) sens_step<SEM & 1>(s[j], or_like, rv[j], rt[j]);
                }
#pragma unroll
                for (int j = 0; j < LW; j++) M[j] &= sens_result<SEM & 1>(s[j]);
            }
        } else if (FIX && (h & RF_MANY) && anyT) {
            // any fan-in may carry the path: its own mark enters the side test
            const uint32_t mor = flagmask(h, RF_IM), mxor = flagmask(h, RF_XOR), mand = ~(mor | mxor);
            SensAcc s[LW];
#pragma unroll
            for (int j = 0; j < LW; j++) sens_init(s[j]);
#pragma unroll
            for (int q = 0; q < kInlineFanins; q++)
                if ((uint32_t)q < nfi)
#pragma unroll
                    for (int j = 0; j < LW; j++)
                        sens_step_fixed<SEM == PDF_MARK_FIXED_NONROBUST>(s[j], mand, mor, mxor, x.fv[q][j],
                                                                         x.ft[q][j], x.fm[q][j]);
            for (uint32_t q = kInlineFanins; q < nfi; q++) {
                uint32_t rv[LW], rt[LW], rm[LW];
                const uint32_t f = far_row(q, rv, rt);
                lzero<LW>(rm);
                if (live && bit_test(bm, f)) lload<LW>(lrow(P.M, f, P.ld4), rm);
#pragma unroll
                for (int j = 0; j < LW; j++)
                    sens_step_fixed<SEM == PDF_MARK_FIXED_NONROBUST>(s[j], mand, mor, mxor, rv[j], rt[j], rm[j]);
            }
#pragma unroll
            for (int j = 0; j < LW; j++) M[j] = T[j] & sens_result<SEM == PDF_MARK_FIXED_NONROBUST>(s[j]);
        }
    }
    const bool marked = MODE != FWD_SIM && __any_sync(0xFFFFFFFFu, lany<LW>(M));
    if (live) {
        if (MODE != FWD_MARK && (a.store_all || (h & RF_SPILL) || marked)) {
            lstore<LW>(lrow(P.V, g, P.ld4), V, nw);
            lstore<LW>(lrow(P.T, g, P.ld4), T, nw);
        }
        if (MODE != FWD_SIM && (a.store_all || marked)) lstore<LW>(lrow(P.M, g, P.ld4), M, nw);
    }
    if (marked && (threadIdx.x & 31) == 0) {
        atomicOr(bm + (g >> 5), 1u << (g & 31));
        if (MODE == FWD_FUSED) atomicMax(reach, rp->w[1] >> 16);
    }
    return marked;
}

// U: gates per warp in flight (their fan-in rows are loaded before any of
// them is evaluated), as many as the registers hold.
template <int SEM, int MODE, int U, int LW>
__device__ __forceinline__ void forward_lanes_cta(const FwdArgs &a, const uint32_t blk) {
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr uint32_t BWL = 32 * LW;                    // words per column block
    constexpr uint32_t NF = BWL / kLaneCoverWords;       // cover bitmaps per block
    constexpr uint32_t SUBL = kLaneCoverWords / LW;      // lanes per cover bitmap
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
    const uint32_t w0 = blk * BWL, w = w0 + lane * LW;
    const bool live = w < a.W;
    const uint32_t nw = live ? min((uint32_t)LW, a.W - w) : 0u;  // words of the lane that hold pairs
    uint32_t wm[LW];
#pragma unroll
    for (int j = 0; j < LW; j++)
        wm[j] = w + j >= a.W ? 0u
                             : (w + j + 1 < a.W ? 0xFFFFFFFFu
                                                : ((a.n_pairs & 31) ? (1u << (a.n_pairs & 31)) - 1u : 0xFFFFFFFFu));
    LanePlanes P;
    P.ld4 = (uint32_t)(a.ld * 4);
    P.V = reinterpret_cast<char *>(a.V + w);
    P.T = reinterpret_cast<char *>(a.T + w);
    P.M = reinterpret_cast<char *>(a.M + w);
    uint32_t *bm = a.bm_shared ? reinterpret_cast<uint32_t *>(smraw + a.off_bm) : a.nzb + (size_t)blk * a.bm_words;
    uint32_t *gbm = a.nzb ? a.nzb + (size_t)blk * a.bm_words : nullptr;
    GateRec *recs = reinterpret_cast<GateRec *>(smraw + a.off_rec);  // [2][a.cap]
    const uint32_t *lo = a.c.level_off;

    if (MODE != FWD_SIM)
        for (uint32_t q = threadIdx.x; q < a.bm_words; q += blockDim.x) bm[q] = 0;
    uint32_t *fine = MODE == FWD_FUSED && a.nzb_fine ? a.nzb_fine + (size_t)blk * NF * a.bm_words : nullptr;
    if (fine)
        for (uint32_t q = threadIdx.x; q < NF * a.bm_words; q += blockDim.x) fine[q] = 0;
    if (MODE == FWD_FUSED) {  // the batch's cover state (the cover kernels run after this one)
        if (a.active && threadIdx.x < BWL && w0 + threadIdx.x <= a.W) a.active[w0 + threadIdx.x] = 0;
        if (a.active && blk == 0 && threadIdx.x == 0) a.active[a.W] = 0;
        if (a.acc && blk == 0 && threadIdx.x == 0) {
            a.acc->batch_lo = 0;
            a.acc->batch_hi = 0;
            a.acc->batch_flags = 0;
            a.acc->done = 0;
            a.acc->n_over = 0;
            a.acc->done_over = 0;
        }
    }
    // the last level that can still hold a marked gate (a lane plan's reach)
    __shared__ uint32_t s_reach;
    const bool early = MODE == FWD_FUSED && a.in_pieces;
    if (threadIdx.x == 0) s_reach = 0;
    __syncthreads();

    // ------------------------------------------------------------- forward
    // Pieces (runs of one level, <= a.cap gates) in level order; the records
    // of each piece are copied into shared memory (cp.async, 16 bytes per
    // thread and copy) while the piece before it is evaluated, and its
    // descriptor is loaded a piece earlier still.  One barrier per piece.
    const auto stage = [&](uint32_t ga, uint32_t gb, int buf) {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.c.rec + ga);
        uint4 *dst = reinterpret_cast<uint4 *>(recs + (size_t)buf * a.cap);
        for (uint32_t i = threadIdx.x; i < 2 * (gb - ga); i += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + i)), "l"(src + i) : "memory");
    };
    // gates [pa, pb) of level pl: the next piece to evaluate; (na, nb, nlv):
    // the one after it, loaded a piece ahead
    uint32_t top = 0;  // levels below `top` may hold a forward mark
    uint32_t pa = a.pieces[0].a, pb = a.pieces[0].b, pl = a.pieces[0].level, na = 0, nb = 0, nlv = 0;
    if (a.n_pieces > 1) {
        na = a.pieces[1].a;
        nb = a.pieces[1].b;
        nlv = a.pieces[1].level;
    }
    stage(pa, pb, 0);
    bool any = false;
    uint32_t prev_level = 0;
    for (uint32_t i = 0; i < a.n_pieces; i++) {
        cp_async_wait_all();  // this thread's copies of piece i's records
        if (__syncthreads_or(any) && i) top = max(top, prev_level + 1);
        any = false;
        // nothing from this level on can be marked (decided where every mark of
        // the levels below is known; s_reach grows only in CTAs that went on)
        if (early && s_reach < pl) break;
        if (i + 1 < a.n_pieces) stage(na, nb, (i + 1) & 1);  // into the buffer of piece i - 1, which every warp has left
        const uint32_t ga = pa, gb = pb;
        prev_level = pl;
        pa = na;
        pb = nb;
        pl = nlv;
        if (i + 2 < a.n_pieces) {
            na = __ldg(&a.pieces[i + 2].a);
            nb = __ldg(&a.pieces[i + 2].b);
            nlv = __ldg(&a.pieces[i + 2].level);
        }
        const GateRec *rb = recs + (size_t)(i & 1) * a.cap;
        for (uint32_t g = ga + warp; g < gb; g += U * NW) {
            LaneIn<LW> x[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t gu = g + u * NW;
                if (gu < gb) lane_load<SEM, MODE, LW>(a, P, bm, rb + (gu - ga), gu, w, live, x[u]);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t gu = g + u * NW;
                if (gu < gb) any |= lane_gate<SEM, MODE, LW>(a, P, bm, rb + (gu - ga), gu, live, nw, wm, &s_reach, x[u]);
            }
        }
    }
    if (__syncthreads_or(any)) top = max(top, prev_level + 1);
    if constexpr (MODE == FWD_SIM) {
        return;
    } else {
        if (MODE == FWD_MARK && a.no_prune) return;
        // ------------------------------------------------- prune and merge
        // (markkernel.cuh:271-293, mergekernel.cuh:116-198) levels descending;
        // a warp takes 32-gate words of the bitmap and visits their marked
        // gates; a gate's pruned mark is final once its fan-outs' are.
        uint32_t maxlvl = 0;
        for (int l = (int)top - 1; l >= 0; l--) {
            const uint32_t ga = __ldg(lo + l), gb = __ldg(lo + l + 1);
            bool any = false;
            for (uint32_t q = (ga >> 5) + warp; q < (gb + 31) >> 5; q += NW) {
                uint32_t bits = bm[q];
                if (q == ga >> 5 && (ga & 31)) bits &= ~((1u << (ga & 31)) - 1u);
                if (q == (gb - 1) >> 5 && (gb & 31)) bits &= (1u << (gb & 31)) - 1u;
                while (bits) {
                    const uint32_t g = q * 32 + (__ffs(bits) - 1);
                    bits &= bits - 1;
                    const GateRec r = load_rec(a.c.rec + g);
                    uint32_t *mrow = lrow(P.M, g, P.ld4);
                    uint32_t mk[LW], keep[LW], nm[LW];
                    lzero<LW>(mk);
                    if (live) lload<LW>(mrow, mk);
#pragma unroll
                    for (int j = 0; j < LW; j++) {
                        mk[j] &= wm[j];  // words past the last pair hold no mark
                        keep[j] = rec_po(r) ? 0xFFFFFFFFu : 0u;
                    }
                    if (!rec_po(r)) {
                        const uint32_t nfo = r.w[1] & a.c.nfo_mask, base = r.w[2] + rec_nfi(r);
                        for (uint32_t k = 0; k < nfo; k += 4) {  // four fan-out rows in flight
                            uint32_t fo[4], m[4][LW];
#pragma unroll
                            for (int u = 0; u < 4; u++) fo[u] = k + u < nfo ? __ldg(a.c.edges + base + k + u) : kEmpty;
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                lzero<LW>(m[u]);
                                if (fo[u] != kEmpty && live && bit_test(bm, fo[u])) lload<LW>(lrow(P.M, fo[u], P.ld4), m[u]);
                            }
#pragma unroll
                            for (int j = 0; j < LW; j++) keep[j] |= m[0][j] | m[1][j] | m[2][j] | m[3][j];
                        }
                    }
                    bool changed = false;
#pragma unroll
                    for (int j = 0; j < LW; j++) {
                        nm[j] = mk[j] & keep[j];
                        changed |= nm[j] != mk[j];
                    }
                    if (live && changed) lstore<LW>(mrow, nm, nw);
                    const uint32_t nzl = __ballot_sync(0xFFFFFFFFu, lany<LW>(nm));  // lanes still marked
                    const bool nz = nzl != 0;
                    if (!nz) {
                        if (lane == 0) atomicAnd(bm + (g >> 5), ~(1u << (g & 31)));
                    } else if (fine && lane < NF && ((nzl >> (SUBL * lane)) & ((1u << SUBL) - 1u))) {
                        atomicOr(fine + (size_t)lane * a.bm_words + (g >> 5), 1u << (g & 31));  // bitmap `lane`
                    }
                    if (nz && MODE == FWD_FUSED && a.first_x) {  // merge: first falling / rising pair
                        uint32_t v[LW];
                        lzero<LW>(v);
                        if (live) lload<LW>(lrow(P.V, g, P.ld4), v);
                        uint32_t cx = kEmpty, cy = kEmpty;
#pragma unroll
                        for (int j = LW - 1; j >= 0; j--) {  // the lowest word last
                            const uint32_t x = nm[j] & ~v[j], y = nm[j] & v[j];
                            if (x) cx = (w + j) * 32 + (__ffs(x) - 1);
                            if (y) cy = (w + j) * 32 + (__ffs(y) - 1);
                        }
                        cx = __reduce_min_sync(0xFFFFFFFFu, cx);
                        cy = __reduce_min_sync(0xFFFFFFFFu, cy);
                        if (lane == 0) {
                            const uint32_t id = net_id(a.c, g);
                            if (cx != kEmpty) atomicMin(a.first_x + id, a.pair_base + cx);
                            if (cy != kEmpty) atomicMin(a.first_y + id, a.pair_base + cy);
                        }
                    }
                    any |= nz;
                }
            }
            if (__syncthreads_or(any) && !maxlvl) maxlvl = (uint32_t)l + 1;
        }
        // publish the bitmap of surviving marks for the cover kernels
        if (a.bm_shared && gbm)
            for (uint32_t q = threadIdx.x; q < a.bm_words; q += blockDim.x) gbm[q] = bm[q];
        if (threadIdx.x == 0) a.blk_maxlvl[blk] = maxlvl;
        if (fine && threadIdx.x < NF) a.maxlvl_fine[blk * NF + threadIdx.x] = maxlvl;
    }
}

// Gates per warp in flight, by tile and semantics (the FIXED modes and the
// stage call pdf_mark carry more rows per gate).  More warps beat more gates
// per warp: on a 1M-gate circuit at 64 words, 1,024 threads with one gate
// each took 36 ms against 46 ms for 512 threads with three or four.
template <int SEM, int MODE, int LW>
struct LaneU {
    static constexpr bool heavy = SEM >= 2 || MODE == FWD_MARK;
    static constexpr int value = LW == 1 ? (heavy ? 2 : 2) : LW == 2 ? (heavy ? 1 : 1) : (heavy ? 1 : 1);
};

template <int SEM, int MODE, int LW>
__global__ void __launch_bounds__(lane_threads(32 * LW), 1) k_forward_lanes(const FwdArgs a) {
    forward_lanes_cta<SEM, MODE, LaneU<SEM, MODE, LW>::value, LW>(a, blockIdx.x);
}

// The same for the circuits of a batch that take a lane tile.
template <int SEM, int LW>
__global__ void __launch_bounds__(lane_threads(32 * LW), 1)
    k_batch_forward_lanes(const FwdArgs *args, const uint32_t *bpref, uint32_t n, BatchCtl *ctl, uint32_t blk0) {
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
    forward_lanes_cta<SEM, FWD_FUSED, LaneU<SEM, FWD_FUSED, LW>::value, LW>(s_a, s_blk);
}


template <int SEM, int MODE, int LW>
cudaError_t launch_t(const FwdArgs &a, uint32_t threads, size_t smem, cudaStream_t st) {
    const uint32_t blocks = (a.W + 32 * LW - 1) / (32 * LW);
    if (blocks == 0 || threads % 32 || threads > lane_threads(32 * LW)) return cudaErrorInvalidValue;
    auto kern = k_forward_lanes<SEM, MODE, LW>;
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <int SEM, int LW>
cudaError_t launch_sem(const FwdArgs &a, int mode, uint32_t threads, size_t smem, cudaStream_t st) {
    switch (mode) {
        case FWD_FUSED: return launch_t<SEM, FWD_FUSED, LW>(a, threads, smem, st);
        case FWD_SIM: return launch_t<SEM, FWD_SIM, LW>(a, threads, smem, st);
        default: return launch_t<SEM, FWD_MARK, LW>(a, threads, smem, st);
    }
}

template <int LW>
cudaError_t launch_lw(const FwdArgs &a, int mode, int sem, uint32_t threads, size_t smem,
                      cudaStream_t st) {
    switch (sem) {
        case 0: return launch_sem<0, LW>(a, mode, threads, smem, st);
        case 1: return launch_sem<1, LW>(a, mode, threads, smem, st);
        case 2: return launch_sem<2, LW>(a, mode, threads, smem, st);
        case 3: return launch_sem<3, LW>(a, mode, threads, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int SEM, int LW>
int regs_lanes_t() {
    cudaFuncAttributes fa{}, fb{};
    if (cudaFuncGetAttributes(&fa, k_forward_lanes<SEM, FWD_FUSED, LW>) != cudaSuccess ||
        cudaFuncGetAttributes(&fb, k_batch_forward_lanes<SEM, LW>) != cudaSuccess) {
        (void)cudaGetLastError();
        return -1;
    }
    return std::max(fa.numRegs, fb.numRegs);
}
template <int LW>
int regs_lanes(int sem) {
    switch (sem) {
        case 0: return regs_lanes_t<0, LW>();
        case 1: return regs_lanes_t<1, LW>();
        case 2: return regs_lanes_t<2, LW>();
        case 3: return regs_lanes_t<3, LW>();
        default: return -1;
    }
}

template <int SEM>
cudaError_t prepare_sem(uint32_t bw, size_t smem) {
    switch (bw) {
        case kLaneWords: return raise_smem_limit(reinterpret_cast<const void *>(k_batch_forward_lanes<SEM, 1>), smem);
        case kLaneWords2: return raise_smem_limit(reinterpret_cast<const void *>(k_batch_forward_lanes<SEM, 2>), smem);
        case kLaneWords4: return raise_smem_limit(reinterpret_cast<const void *>(k_batch_forward_lanes<SEM, 4>), smem);
        default: return cudaErrorInvalidValue;
    }
}
template <int SEM>
cudaError_t launch_class_sem(const BatchLaunch &b, const BatchClass &c, cudaStream_t s) {
    switch (c.bw) {
        case kLaneWords:
            k_batch_forward_lanes<SEM, 1><<<c.blocks, c.threads, c.smem, s>>>(b.fargs, b.bpref, b.n, b.ctl, c.blk0);
            break;
        case kLaneWords2:
            k_batch_forward_lanes<SEM, 2><<<c.blocks, c.threads, c.smem, s>>>(b.fargs, b.bpref, b.n, b.ctl, c.blk0);
            break;
        case kLaneWords4:
            k_batch_forward_lanes<SEM, 4><<<c.blocks, c.threads, c.smem, s>>>(b.fargs, b.bpref, b.n, b.ctl, c.blk0);
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace

int lane_kernel_regs(int bw, int sem) {
    switch (bw) {
        case kLaneWords: return regs_lanes<1>(sem);
        case kLaneWords2: return regs_lanes<2>(sem);
        case kLaneWords4: return regs_lanes<4>(sem);
        default: return -1;
    }
}

cudaError_t launch_lanes(const FwdArgs &a, int mode, int sem, uint32_t bw, uint32_t threads,
                         size_t smem, cudaStream_t st) {
    switch (bw) {
        case kLaneWords: return launch_lw<1>(a, mode, sem, threads, smem, st);
        case kLaneWords2: return launch_lw<2>(a, mode, sem, threads, smem, st);
        case kLaneWords4: return launch_lw<4>(a, mode, sem, threads, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t prepare_lanes_class(uint32_t sem, uint32_t bw, size_t smem) {
    switch (sem) {
        case 0: return prepare_sem<0>(bw, smem);
        case 1: return prepare_sem<1>(bw, smem);
        case 2: return prepare_sem<2>(bw, smem);
        case 3: return prepare_sem<3>(bw, smem);
        default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_lanes_class(const BatchLaunch &b, const BatchClass &c, cudaStream_t s) {
    switch (b.sem) {
        case 0: return launch_class_sem<0>(b, c, s);
        case 1: return launch_class_sem<1>(b, c, s);
        case 2: return launch_class_sem<2>(b, c, s);
        case 3: return launch_class_sem<3>(b, c, s);
        default: return cudaErrorInvalidValue;
    }
}
