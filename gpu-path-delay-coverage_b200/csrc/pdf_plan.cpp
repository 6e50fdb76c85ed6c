// pdf_plan.cpp -- launch plans of the forward kernels (host code).
#include "pdf_plan.h"

#include <algorithm>

#include "pdf_kernels.cuh"

void build_records(const NetPlan &n, LaunchPlan &pl) {
    const uint32_t G = n.n_gates();
    pl.n_gates = G;
    pl.n_levels = n.n_levels();
    pl.nfo_mask = 0xFFFFFFFFu;
    pl.recs.assign(G, GateRec{});
    for (uint32_t g = 0; g < G; g++) {
        GateRec &r = pl.recs[g];
        r.w[0] = n.hdr[g];
        r.w[1] = n.nfo[g];
        r.w[2] = (uint32_t)n.eoff[g];  // w[3..6]: source words, set below
        // fan-in 0; of an input, its row in the pair planes
        r.w[7] = n.nfi[g] ? n.edges[n.eoff[g]] : (n.hdr[g] & RF_INPT ? (n.orig.empty() ? g : n.orig[g]) : 0u);
    }
}

ResidentImage build_resident(const NetPlan &n, size_t smem) {
    ResidentImage im;
    const uint32_t G = n.n_gates(), L = n.n_levels();
    if (G > 0xFFFFu || L > 0xFFFFu || (size_t)G * 28 > smem) return im;
    uint64_t n_edge = 0;
    for (uint32_t g = 0; g < G; g++) n_edge += n.nfo[g] + (n.nfi[g] > kInlineFanins ? n.nfi[g] : 0);
    if (n_edge > 0xFFFFu) return im;
    const auto a16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t o_edge = 16 * ((size_t)G + 1), o_lvl = o_edge + a16(2 * n_edge), o_ids = o_lvl + 8 * ((size_t)L + 1);
    // one word per block at least, and the ids where there is room for them
    const size_t words = (size_t)G * 12 + a16((G + 31) / 32 * 4) + 128;
    if (a16(o_ids) + words > smem) return im;
    im.ids = a16(o_ids + 4 * (size_t)G) + words <= smem;
    const size_t total = a16(o_ids + (im.ids ? 4 * (size_t)G : 0));
    // how far each gate's mark reaches: the last level of the gates it carries to
    std::vector<uint16_t> reach(G, 0);
    for (uint32_t l = 0; l < L; l++)
        for (uint32_t g = n.level_off[l]; g < n.level_off[l + 1]; g++) {
            const uint32_t *fin = n.edges.data() + n.eoff[g];
            if (n.hdr[g] & RF_MANY)
                for (uint32_t q = 0; q < n.nfi[g]; q++) reach[fin[q]] = (uint16_t)l;
            else if ((n.hdr[g] & RF_MARKF0) && n.nfi[g])
                reach[fin[0]] = (uint16_t)l;
        }
    im.bytes.assign(total, 0);
    im.off_edge = (uint32_t)o_edge;
    im.off_lvl = (uint32_t)o_lvl;
    uint32_t *rec = reinterpret_cast<uint32_t *>(im.bytes.data());
    uint16_t *edge = reinterpret_cast<uint16_t *>(im.bytes.data() + o_edge);
    uint32_t *lvl = reinterpret_cast<uint32_t *>(im.bytes.data() + o_lvl), at = 0;
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t *e = n.edges.data() + n.eoff[g], nfi = n.nfi[g];
        uint32_t *r = rec + 4 * (size_t)g, f[4] = {0, 0, 0, 0};
        for (uint32_t q = 0; q < nfi && q < 4; q++) f[q] = e[q];
        r[0] = n.hdr[g];
        r[1] = f[0] | f[1] << 16;
        r[2] = f[2] | f[3] << 16;
        if (n.hdr[g] & RF_INPT) r[1] = n.orig.empty() ? g : n.orig[g];
        r[3] = at | (uint32_t)reach[g] << 16;
        for (uint32_t q = nfi > kInlineFanins ? 0 : nfi; q < nfi + n.nfo[g]; q++) edge[at++] = (uint16_t)e[q];
    }
    rec[4 * (size_t)G + 3] = at;
    for (uint32_t g = 0; im.ids && g < G; g++) lvl[2 * ((size_t)L + 1) + g] = n.orig.empty() ? g : n.orig[g];
    for (uint32_t l = 0; l <= L; l++) {
        lvl[2 * l] = n.level_off[l];
        // gates up to the last that marks (a reduced netlist lists those first)
        if (l < L)
            for (uint32_t g = n.level_off[l]; g < n.level_off[l + 1]; g++)
                if (n.hdr[g] & (RF_MARKF0 | RF_MANY)) lvl[2 * l + 1] = g + 1 - n.level_off[l];
    }
    return im;
}

// Column block and CTAs of a resident walk over W words: the block width with
// the least modelled time.  A block costs its level chain (forward and prune,
// about 0.3 us a level, of as many blocks at once as CTAs fit an SM) or its
// instructions (about 0.42 ns per gate and word of an SM), whichever is more;
// a CTA the copy of the image first, shared by the blocks it takes in turn.
// With plane rows every gate also stores a piece of each, a sector whatever the
// block's width: 5.5 ns a gate for three, 3.2 for two, and all levels are walked.
ResidentShape resident_shape(const ResidentSizes &z, uint64_t W, uint32_t rows) {
    const auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    ResidentShape best;
    uint32_t words = 0;
    for (uint32_t bw = 1; bw <= 8; bw *= 2) {
        ResidentShape s;
        s.bw = bw;
        size_t off = al(z.image_bytes);
        s.off_vt = (uint32_t)off;
        off += 8 * (size_t)bw * z.n_gates;
        s.off_m = (uint32_t)off;
        off = al(off + 4 * (size_t)bw * z.n_gates);
        s.off_bm = (uint32_t)off;
        off = al(off + ((size_t)z.n_gates + 31) / 32 * 4);
        s.off_mbar = (uint32_t)off;
        s.smem = off + 16;
        if (s.smem + 1024 > z.smem_block) break;  // (and the kernels' static variables)
        const uint32_t by_smem = (uint32_t)std::max<size_t>(1, z.smem_sm / (s.smem + 2048));
        s.threads = by_smem >= 2 ? 256 : 512;
        s.occ = std::min({by_smem, 2048 / s.threads, 65536 / (s.threads * std::max(z.regs, 32u)), 8u});
        while (s.occ & (s.occ - 1)) s.occ &= s.occ - 1;  // 1, 2, 4 or 8: few classes in a batch
        words = std::max(words, s.occ * bw);
        s.blocks = (uint32_t)((W + bw - 1) / bw);
        const uint32_t slots = z.sms * s.occ;
        s.per = (s.blocks + slots - 1) / slots;
        s.ctas = (s.blocks + s.per - 1) / s.per;
        const double load = 2.0 + z.image_bytes / 95e3;
        const uint32_t together = std::min(s.occ, (s.ctas + z.sms - 1) / z.sms);
        const double issue = 0.42e-3 * z.n_gates * bw;
        if (rows) {
            const double chain = rows == 3 ? 4.0 + 0.25 * z.n_levels : 3.0 + 0.2 * z.n_levels;
            const double stores = (rows == 3 ? 5.5e-3 : 3.2e-3) * z.n_gates;
            s.us = load + s.per * (chain + together * (stores + issue));
        } else {
            const double chain = 1.0 + 0.3 * z.n_levels;
            s.block_us = std::max(chain / s.occ, issue);
            s.us = load + s.per * std::max(chain, together * issue);
        }
        if (!best.bw || s.us < best.us * 0.97) best = s;
    }
    best.words = words;
    return best;
}

// A round of blocks costs about 0.4 of the staged kernel's walk, whose CTAs take
// about 10 words an SM at a time: where an SM has room for fewer, two rounds pay.
// Measured (kernels, us, resident and staged; 7,182 gates, 1 word an SM): 256 words
// 56 and 74, 512 words 108 and 81, 2,048 words 339 and 111, 32,768 words 4,988 and
// 1,433; 4,191 gates, 2 words: 512 words 48 and 81, 2,048 words 159 and 103 (FIXED
// 384 and 239); 3,159 gates, 4 words: 512 words 20 and 68, 2,048 words 71 and 68,
// 8,192 words 236 and 160; 1,554 gates, 8 words: 8,192 words 112 and 154, 32,768
// words 418 and 492.
uint64_t resident_words(const ResidentShape &s, uint32_t sms) {
    return s.words >= kResidentWords ? ~0ull : 2ull * s.words * sms;
}
bool resident_pays(const ResidentShape &s, uint64_t W, uint32_t sms) { return W <= resident_words(s, sms); }

// The staged kernel walks all gates: about 1 us a piece and 11 ps a gate and
// word (6.5 ps the codes alone).  Narrow blocks stop paying where rows are long
// for another reason: the sectors that a CTA has written a part of leave L2
// before its next blocks fill them.  Measured (kernels, us, resident with the
// fill beside it, and staged; all planes / codes alone): 5,300 gates that all
// switch, 150 levels: 256 words 143 / 104 and 225 / 168, 1,024 words 481 / 342 and
// 280 / 181, 2,048 words 952 / 674 and 306 / 199; 2,500 gates, 60 levels: 1,024
// words 79 / 56 and 124 / 74, 2,048 words 145 / 104 and 137 / 83; 20,000 gates,
// 3,367 not constant: 2,048 words 258 / 162 and 551 / 329, 8,192 words 1,838 / 1,532
// and 1,904 / 1,207; 26,000 gates, 4,400 not constant: 1,024 words 282 / 185 and
// 569 / 267, 4,955 words 4,320 and 2,498.
bool resident_planes_pay(const ResidentShape &s, uint64_t W, uint32_t rows, uint64_t gates, uint32_t pieces) {
    if (W > 1024ull * s.bw * s.bw) return false;
    const double cells = (double)gates * W;
    const double staged = rows == 3 ? 40.0 + 1.05 * pieces + 11e-6 * cells : 10.0 + 0.95 * pieces + 6.5e-6 * cells;
    return 1.15 * (s.us + 5.0) <= staged;  // (and the fill's launch)
}

pdf_status build_plan(const NetPlan &n, const PlanOpts &o, LaunchPlan &pl) {
    const uint32_t G = n.n_gates(), L = n.n_levels();
    uint32_t widest_level = 0;
    for (uint32_t l = 0; l < L; l++) widest_level = std::max(widest_level, n.level_off[l + 1] - n.level_off[l]);
    build_records(n, pl);
    pl.bw = o.bw;
    const bool lanes = lane_tile(pl.bw);
    if (lanes) {
        // The lane kernel reads every fan-in from its plane row: source words
        // are the fan-in ids themselves, flagged SRC_ZERO when the fan-in is
        // a killed gate (S0 whatever its inputs); a gate writes its rows
        // (RF_SPILL) only when some gate reads them.
        std::vector<uint8_t> read(G, 0);
        for (uint32_t g = 0; g < G; g++)
            for (uint32_t q = 0; q < n.nfi[g]; q++) {
                const uint32_t f = n.edges[n.eoff[g] + q];
                const bool zero = q < kInlineFanins && (pl.recs[f].w[0] & RF_KILL) && !(pl.recs[f].w[0] & RF_OINV);
                if (q < kInlineFanins) pl.recs[g].w[3 + q] = f | (zero ? SRC_ZERO : 0u);
                if (!zero) read[f] = 1;
            }
        for (uint32_t g = 0; g < G; g++)
            if (read[g]) pl.recs[g].w[0] |= RF_SPILL;
    }
    const uint32_t max_threads = lanes ? lane_threads(pl.bw) : (pl.bw >= 8 ? 512 : 1024);
    uint32_t threads_default = 512;  // set from the piece size below
    auto al = [](size_t x) { return (x + 127) & ~(size_t)127; };
    const uint32_t bm_words = (G + 31) / 32;
    // Pieces (the kernels' unit of staging and of synchronisation), sized
    // from the widest level above the inputs (the inputs' level, often the
    // widest, just splits into more pieces): runs of one level, <= cap gates,
    // edge slice <= ecap words.
    uint32_t widest = 1;
    for (uint32_t l = 1; l < L; l++) widest = std::max(widest, n.level_off[l + 1] - n.level_off[l]);
    if (L == 1) widest = widest_level;
    pl.cap = lanes ? 0u : std::min<uint32_t>(512, (widest + 31) & ~31u);
    // one thread per gate of a piece plus two warps that have none: they
    // issue the next piece's far-row copies
    threads_default = lanes ? lane_threads(pl.bw) : std::min<uint32_t>(max_threads, pl.cap + 64);
    pl.threads = o.threads ? std::min(o.threads, max_threads) : threads_default;
    // a block size given by the caller also bounds the pieces: threads - 64
    // gates, so two warps stay free for the far-row copies
    if (!lanes && o.threads && pl.threads >= 128) pl.cap = std::min(pl.cap, (pl.threads - 64) & ~31u);
    // CTAs per SM that the registers allow for this block size (at most 4);
    // the dynamic shared memory of the forward kernels is then an equal share
    // of the SM, less 1 KiB per CTA the system keeps and 1 KiB for the
    // kernels' static variables (the batched kernel keeps its arguments there).
    {
        if (o.regs <= 0) return PDF_ECUDA;
        const uint32_t warps = (pl.threads + 31) / 32;
        const uint32_t warp_regs = ((uint32_t)o.regs * 32 + 255) & ~255u;
        uint32_t occ = std::min<uint32_t>(65536 / (warps * warp_regs), 2048 / (warps * 32));
        pl.occ = std::max<uint32_t>(1, std::min<uint32_t>(occ, 4));
    }
    const size_t budget = std::min<size_t>((size_t)o.smem_block,
                                           (size_t)o.smem_sm / pl.occ - 1024) -
                          1024;
    pl.ecap = 2048;
    if (lanes) {
        // The lane kernel keeps on chip two buffers of staged gate records
        // and the column block's mark bitmap (in global memory when it does
        // not fit); its pieces are runs of one level of <= cap gates: 2 x
        // kLaneRecs when those buffers fit beside a shared-memory bitmap (a
        // barrier per piece, so wide levels take half as many), else
        // kLaneRecs.
        const size_t bm_bytes = (size_t)bm_words * 4;
        pl.cap = kLaneRecs;
        if (widest > kLaneRecs &&
            2 * 2 * (size_t)kLaneRecs * sizeof(GateRec) + al(bm_bytes) + 2048 <= budget)
            pl.cap = 2 * kLaneRecs;
        for (uint32_t l = 0; l < L; l++)
            for (uint32_t a = n.level_off[l]; a < n.level_off[l + 1]; a += pl.cap) {
                Piece p{};
                p.a = a;
                p.b = std::min(a + pl.cap, n.level_off[l + 1]);
                p.level = l;
                pl.pieces.push_back(p);
            }
        pl.n_pieces = (uint32_t)pl.pieces.size();
        const size_t rec_bytes = 2 * (size_t)pl.cap * sizeof(GateRec);
        pl.off_rec = 0;
        pl.off_bm = (uint32_t)rec_bytes;
        pl.bm_shared = rec_bytes + bm_bytes + 2048 <= budget ? 1u : 0u;
        pl.fwd_smem = rec_bytes + (pl.bm_shared ? al(bm_bytes) : 0);
        pl.chain = G;
        while (pl.far_ids.size() < 4) pl.far_ids.push_back(0);
    } else {
        auto f4 = [](uint64_t x) { return x & ~(uint64_t)3; };
        auto c4 = [](uint64_t x) { return (x + 3) & ~(uint64_t)3; };
        for (uint32_t l = 0; l < L; l++) {
            const uint32_t s0 = n.level_off[l], e0 = n.level_off[l + 1];
            for (uint32_t a = s0; a < e0;) {
                uint32_t b = a + 1;
                while (b < e0 && b - a < pl.cap && c4(n.eoff[b + 1]) - f4(n.eoff[a]) <= pl.ecap) b++;
                Piece p{};
                p.a = a;
                p.b = b;
                p.level = l;
                if (c4(n.eoff[b]) - f4(n.eoff[a]) <= pl.ecap) {
                    p.ea = (uint32_t)f4(n.eoff[a]);
                    p.eb = (uint32_t)c4(n.eoff[b]);
                } else {
                    p.ea = p.eb = 0xFFFFFFFFu;  // one gate with a huge edge list: read in place
                }
                pl.pieces.push_back(p);
                a = b;
            }
        }
        pl.n_pieces = (uint32_t)pl.pieces.size();
        if (pl.n_pieces > 65536) return PDF_ENOTSUP;
        // Far fan-ins of piece i (ring of R slots): fan-ins 0..3 of its gates
        // below b_i - R.  Those below a_{i-1} (complete when piece i - 1 starts)
        // go to the piece's deduplicated far list, up to `limit` entries; the rest
        // are read from their plane rows.  Fills the source words w[3..6].
        auto far_lists = [&](uint32_t R, uint32_t limit) -> uint32_t {
            uint32_t worst = 0;
            pl.far_ids.clear();
            std::vector<uint32_t> seen(G, 0xFFFFFFFFu);  // gate -> slot in the current piece's list
            std::vector<uint32_t> list;
            for (size_t i = 0; i < pl.pieces.size(); i++) {
                Piece &p = pl.pieces[i];
                const uint32_t lo = p.b > R ? p.b - R : 0;
                const uint32_t done = i ? pl.pieces[i - 1].a : 0;
                list.clear();
                for (uint32_t g = p.a; g < p.b; g++) {
                    const uint32_t nq = std::min<uint32_t>(n.nfi[g], kInlineFanins);
                    for (uint32_t q = 0; q < nq; q++) {
                        const uint32_t f = n.edges[n.eoff[g] + q];
                        uint32_t sw = f & (R - 1);
                        if (f < lo) {
                            sw = SRC_PLANE | f;
                            if (f < done) {
                                if (seen[f] == 0xFFFFFFFFu && list.size() < limit) {
                                    seen[f] = (uint32_t)list.size();
                                    list.push_back(f);
                                }
                                if (seen[f] != 0xFFFFFFFFu) sw = SRC_FAR | seen[f];
                            }
                        }
                        pl.recs[g].w[3 + q] = sw;
                        if (sw & SRC_PLANE || sw & SRC_FAR) pl.recs[f].w[0] |= RF_SPILL;
                    }
                    for (uint32_t q = kInlineFanins; q < n.nfi[g]; q++) {  // read from edges[] at run time
                        const uint32_t f = n.edges[n.eoff[g] + q];
                        if (f < lo) pl.recs[f].w[0] |= RF_SPILL;
                    }
                }
                for (uint32_t f : list) seen[f] = 0xFFFFFFFFu;
                worst = std::max<uint32_t>(worst, (uint32_t)list.size());
                p.far_off = (uint32_t)pl.far_ids.size();
                p.far_n = (uint32_t)list.size();
                pl.far_ids.insert(pl.far_ids.end(), list.begin(), list.end());
                // lists start on 16-byte boundaries: the kernel stages the next
                // piece's list by a bulk copy located from this piece's fields
                while (pl.far_ids.size() & 3) pl.far_ids.push_back(0);
            }
            for (size_t i = 0; i < pl.pieces.size(); i++) pl.pieces[i].nfar_n = i + 1 < pl.pieces.size() ? pl.pieces[i + 1].far_n : 0;
            return worst;
        };
        // Shared memory of k_forward: 2 record buffers; one region holding the
        // reverse pass's 2 edge buffers or the forward pass's 2 far buffers;
        // bitmap; piece bits; barriers; the ring.  The ring: the largest power of
        // two (>= cap, <= 2 * n_gates) that leaves room for far lists of 64
        // entries; the far lists then get the rest of the budget.
        const size_t rec_bytes = al(2 * (size_t)pl.cap * sizeof(GateRec));
        const size_t bm_bytes = (size_t)bm_words * 4 <= 16384 ? al((size_t)bm_words * 4) : 0;
        const size_t fixed = rec_bytes + bm_bytes + al(((size_t)pl.n_pieces + 31) / 32 * 4) + 128;
        const size_t edge_bytes = 2 * (size_t)pl.ecap * 4;
        const size_t far_entry = (size_t)2 * 3 * pl.bw * 4;  // one far slot in both buffers, 3 planes
        uint32_t rmin = 32;
        while (rmin < pl.cap) rmin *= 2;
        uint32_t rmax = rmin;
        while ((uint64_t)rmax < 2 * (uint64_t)G && fixed + (size_t)rmax * 2 * pl.bw * 12 <= budget) rmax *= 2;
        // the ring's memory also holds the reverse pass's row staging buffers
        const size_t rows_bytes = (size_t)2 * pl.cap * 2 * pl.bw * 4;
        auto ring_bytes = [&](size_t R) { return std::max(R * pl.bw * 12, rows_bytes); };
        // The largest ring that fits wins: a smaller ring with longer far lists
        // was measured slower (1M gates, 5,000-gate levels: 116.8 against 109.9
        // ms) although it leaves fewer fan-ins to plane-row reads.
        // far region (far rows of two pieces, or the reverse pass's edges) and
        // the two staged far-id lists, for lists of n entries
        auto far_bytes = [&](size_t n) { return al(std::max(edge_bytes, n * far_entry)) + al(2 * n * 4); };
        uint32_t ring = 0;
        for (uint32_t R = rmax; R >= rmin && !ring; R /= 2)
            if (fixed + far_bytes(64) + ring_bytes(R) <= budget) ring = R;
        if (!ring) return PDF_ENOTSUP;
        const size_t far_room = budget - fixed - ring_bytes(ring);
        uint32_t far_limit = (uint32_t)std::min<size_t>(kMaxFar, far_room / (far_entry + 8)) & ~3u;
        while (far_limit > 64 && far_bytes(far_limit) > far_room) far_limit -= 4;
        const uint32_t farcap = std::max<uint32_t>(4, (far_lists(ring, far_limit) + 3) & ~3u);
        while (pl.far_ids.size() < 4) pl.far_ids.push_back(0);
        pl.ring = ring;
        pl.farcap = farcap;
        size_t off = 0;
        pl.off_rec = (uint32_t)off;
        off += rec_bytes;
        pl.off_edge = (uint32_t)off;
        off += al(std::max(edge_bytes, farcap * far_entry));
        pl.off_fid = (uint32_t)off;
        off += al(2 * (size_t)farcap * 4);
        pl.bm_shared = bm_bytes ? 1u : 0u;
        pl.off_bm = (uint32_t)off;
        off += bm_bytes;
        pl.off_pbits = (uint32_t)off;
        off += al(((size_t)pl.n_pieces + 31) / 32 * 4);
        pl.off_mbar = (uint32_t)off;
        off += 128;
        pl.off_ring = (uint32_t)off;
        // reverse pass: ring2 and the row staging buffers [2][cap][2][bw] share
        // the ring's memory
        uint32_t ring2 = 0;
        for (uint32_t r = 1; (size_t)r * pl.bw * 4 + rows_bytes <= ring_bytes(ring); r *= 2) ring2 = r;
        pl.ring2 = ring2;
        pl.fwd_smem = off + ring_bytes(ring);
        pl.chain = pl.n_pieces;
    }
    // How far a gate's mark can reach: the last piece (of a lane plan, level)
    // that holds a gate whose mark this one can carry.  Kept above the fan-out count in w[1] where
    // both fit 16 bits; else the walk never ends early.
    pl.nfo_mask = 0xFFFFFFFFu;
    const uint32_t max_nfo = n.nfo.empty() ? 0 : *std::max_element(n.nfo.begin(), n.nfo.end());
    if (max_nfo <= 0xFFFFu && pl.n_pieces <= 0xFFFFu && L <= 0xFFFFu) {
        pl.nfo_mask = 0xFFFFu;
        while (pl.in_pieces < pl.n_pieces && pl.pieces[pl.in_pieces].level == 0) pl.in_pieces++;
        std::vector<uint16_t> reach(G, 0);
        const auto at = [&](uint32_t i) { return (uint16_t)(lanes ? pl.pieces[i].level : i); };
        for (uint32_t i = 0; i < pl.n_pieces; i++)  // ascending: the last reader's piece stays
            for (uint32_t g = pl.pieces[i].a; g < pl.pieces[i].b; g++) {
                const uint32_t *fin = n.edges.data() + n.eoff[g];
                if (n.hdr[g] & RF_MANY)
                    for (uint32_t q = 0; q < n.nfi[g]; q++) reach[fin[q]] = at(i);
                else if ((n.hdr[g] & RF_MARKF0) && n.nfi[g])
                    reach[fin[0]] = at(i);
            }
        for (uint32_t g = 0; g < G; g++) pl.recs[g].w[1] |= (uint32_t)reach[g] << 16;
    }
    return PDF_OK;
}
