// pdf_reduce.h -- what a grading call without plane outputs has to evaluate.
//
// Such a call returns first-detecting pairs and a path count, and both come
// from nets that hold a mark after the prune.  From the netlist alone:
//
//   constant   the value is the same for every pair (a killed gate is S0:
//              the reference's fold sends a multi-input XOR, XNOR or NOT to
//              0, simkernel.cuh:89-92, and what that fixes downstream is
//              fixed too): it never transitions, so it never marks;
//   markable   an input, or a gate that is not constant whose mark-carrying
//              fan-in (fan-in 0; any fan-in in the FIXED modes) is markable
//              (markkernel.cuh:233-264);
//   observable markable, and an output or the fan-in of an observable gate:
//              the nets the prune can leave marked (markkernel.cuh:271-293).
//              Marks of other nets reach no observable net (whose carrying
//              fan-ins are all observable when markable), so they need not
//              be formed at all;
//   needed     observable, or in the fan-in cone of a needed gate that is
//              not constant: its value enters an observable net's mark.
//
// Everything else can be left out of the walk whatever the pairs are.  The
// reduced netlist holds the needed gates that are not constant, renumbered by
// (level, kind of gate, id): levels are longest paths from the inputs over
// the gates that are left, and gates of one kind stand together so that the
// threads of a warp take the same branches.  Constants read by them become
// two pseudo gates (S0 and S1) at the end of level 0.
#ifndef PDF_REDUCE_H
#define PDF_REDUCE_H

#include <algorithm>
#include <cstdint>
#include <vector>

#include "pdf.h"
#include "pdf_device.cuh"

// A netlist in the kernels' form: gates in level order, canonical edges (each
// gate's fan-ins then fan-outs, gates in id order).
struct NetPlan {
    std::vector<uint32_t> level_off;  // [levels + 1]
    std::vector<uint32_t> hdr;        // record header per gate
    std::vector<uint32_t> nfi, nfo;
    std::vector<uint64_t> eoff;       // [gates + 1]
    std::vector<uint32_t> edges;
    std::vector<uint32_t> orig;       // reduced netlists: the caller's gate id (~0: a constant)
    uint32_t n_gates() const { return (uint32_t)hdr.size(); }
    uint32_t n_levels() const { return (uint32_t)level_off.size() - 1; }
};

// The caller's netlist in that form; `fixed`: the true n-input semantics.
inline NetPlan net_plan(const pdf_netlist *nl, bool fixed) {
    NetPlan n;
    const uint32_t G = nl->n_gates;
    n.level_off.assign(nl->level_offsets, nl->level_offsets + nl->n_levels + 1);
    n.nfi.assign(nl->nfi, nl->nfi + G);
    n.nfo.assign(nl->nfo, nl->nfo + G);
    n.hdr.resize(G);
    n.eoff.resize(G + 1);
    n.edges.reserve(nl->n_edges);
    for (uint32_t g = 0; g < G; g++) {
        n.hdr[g] = make_rec_header(nl->type[g], nl->po[g], nl->nfi[g], fixed);
        n.eoff[g] = n.edges.size();
        const uint32_t *e = nl->edges + nl->edge_offset[g];
        n.edges.insert(n.edges.end(), e, e + nl->nfi[g] + nl->nfo[g]);
    }
    n.eoff[G] = n.edges.size();
    return n;
}

struct NetFacts {
    std::vector<int8_t> value;        // 0 or 1: constant under both vectors; -1: not constant
    std::vector<uint8_t> observable;  // can hold a mark after the prune
    std::vector<uint8_t> needed;      // to be evaluated (never a constant)
    uint64_t n_needed = 0;
};

// Three-valued value of a gate from its fan-ins' (-1 = unknown), by the fold
// of eval_first / eval_fold / eval_finish.
inline int const_value(uint32_t h, uint32_t nfi, const uint32_t *fin, const int8_t *val, bool fixed) {
    if (h & RF_INPT) return -1;
    if (h & RF_KILL) return (h & RF_OINV) ? 1 : 0;
    if (!nfi) return 0;
    const auto inv = [](int v, bool x) { return v < 0 || !x ? v : 1 - v; };
    const bool im = h & RF_IM, om = h & RF_OM, x = fixed && (h & RF_XOR);
    int v = inv(val[fin[0]], h & RF_NOT);
    for (uint32_t q = 1; q <= hdr_nfold(h); q++) {
        const int r = val[fin[q]];
        if (x) {
            v = v < 0 || r < 0 ? -1 : v ^ r;
        } else {
            const int a = inv(v, im), b = inv(r, im);
            const int both = a == 0 || b == 0 ? 0 : (a == 1 && b == 1 ? 1 : -1);
            v = inv(both, im != om);
        }
    }
    return inv(v, fixed && (h & RF_OINV));
}

inline NetFacts net_facts(const NetPlan &n, bool fixed) {
    const uint32_t G = n.n_gates();
    NetFacts f;
    f.value.assign(G, -1);
    f.observable.assign(G, 0);
    f.needed.assign(G, 0);
    std::vector<uint8_t> markable(G, 0);
    // (constants come from killed gates and gates without fan-ins alone)
    bool constants = false;
    for (uint32_t g = 0; g < G && !constants; g++)
        constants = (n.hdr[g] & RF_KILL) || (!n.nfi[g] && !(n.hdr[g] & RF_INPT));
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t h = n.hdr[g], *fin = n.edges.data() + n.eoff[g];
        if (constants) f.value[g] = (int8_t)const_value(h, n.nfi[g], fin, f.value.data(), fixed);
        if (f.value[g] >= 0) continue;
        bool m = h & RF_INPT;
        if (!m && (h & RF_MARKF0)) m = markable[fin[0]];
        if (!m && (h & RF_MANY))
            for (uint32_t q = 0; q < n.nfi[g]; q++) m |= markable[fin[q]] != 0;
        markable[g] = m;
    }
    // descending: a gate's fan-outs are on higher levels, so they are done
    for (uint32_t g = G; g-- > 0;) {
        const uint32_t h = n.hdr[g], *e = n.edges.data() + n.eoff[g];
        if (markable[g]) {
            bool o = (h >> 4) & 1u;
            for (uint32_t k = 0; k < n.nfo[g] && !o; k++) o = f.observable[e[n.nfi[g] + k]];
            f.observable[g] = o;
        }
        if (f.observable[g]) f.needed[g] = 1;
        if (!f.needed[g]) continue;
        f.n_needed++;
        for (uint32_t q = 0; q < n.nfi[g]; q++)
            if (f.value[e[q]] < 0) f.needed[e[q]] = 1;
    }
    return f;
}

inline NetPlan reduce_net(const NetPlan &n, const NetFacts &f) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    const uint32_t G = n.n_gates();
    // longest-path levels of the gates that stay
    std::vector<uint32_t> lvl(G, 0);
    uint32_t L = 1;
    for (uint32_t g = 0; g < G; g++) {
        if (!f.needed[g] || (n.hdr[g] & RF_INPT)) continue;
        const uint32_t *fin = n.edges.data() + n.eoff[g];
        uint32_t l = 0;
        for (uint32_t q = 0; q < n.nfi[g]; q++)
            if (f.value[fin[q]] < 0) l = std::max(l, lvl[fin[q]]);
        lvl[g] = l + 1;
        L = std::max(L, l + 2);
    }
    NetPlan r;
    const uint32_t N = (uint32_t)f.n_needed + 2;  // and the two constants
    r.level_off.assign(L + 1, 0);
    for (uint32_t g = 0; g < G; g++)
        if (f.needed[g]) r.level_off[lvl[g] + 1]++;
    r.level_off[1] += 2;
    for (uint32_t l = 0; l < L; l++) r.level_off[l + 1] += r.level_off[l];
    // by level, then by kind (observable first, fan-in count, evaluation
    // flags), then by id: a counting sort by level, then one by kind within
    // each level (a plain sort where the level is much narrower than the buckets)
    constexpr uint32_t kKinds = 512;
    const auto kind = [&](uint32_t g) {
        const uint32_t h = n.hdr[g];
        return (f.observable[g] ? 0u : 256u) | std::min<uint32_t>(n.nfi[g], 4) << 5 |
               ((h >> 16) & 7u) << 2 | ((h & RF_XOR) ? 2u : 0u) | ((h & RF_OINV) ? 1u : 0u);
    };
    struct Entry {
        uint32_t g, kind;
    };
    std::vector<uint32_t> at(r.level_off.begin(), r.level_off.end() - 1);
    std::vector<Entry> sorted(N, Entry{kNone, 0});
    for (uint32_t g = 0; g < G; g++)
        if (f.needed[g]) sorted[at[lvl[g]]++] = Entry{g, kind(g)};
    r.orig.assign(N, kNone);
    uint32_t start[kKinds + 1];
    for (uint32_t l = 0; l < L; l++) {
        const uint32_t o = r.level_off[l], w = at[l] - o;
        Entry *e = sorted.data() + o;
        if (w < 64) {  // (few of a kind apart: by insertion)
            for (uint32_t i = 1; i < w; i++) {
                const Entry x = e[i];
                uint32_t k = i;
                for (; k && e[k - 1].kind > x.kind; k--) e[k] = e[k - 1];
                e[k] = x;
            }
            for (uint32_t i = 0; i < w; i++) r.orig[o + i] = e[i].g;
            continue;
        }
        std::fill(start, start + kKinds + 1, 0u);
        for (uint32_t i = 0; i < w; i++) start[e[i].kind + 1]++;
        for (uint32_t k = 0; k < kKinds; k++) start[k + 1] += start[k];
        for (uint32_t i = 0; i < w; i++) r.orig[o + start[e[i].kind]++] = e[i].g;
    }
    std::vector<uint32_t> id(G, kNone);
    for (uint32_t k = 0; k < N; k++)
        if (r.orig[k] != kNone) id[r.orig[k]] = k;
    const uint32_t c0 = r.level_off[1] - 2;  // S0, then S1
    r.hdr.resize(N);
    r.nfi.assign(N, 0);
    r.nfo.assign(N, 0);
    r.eoff.assign(N + 1, 0);
    uint64_t most = 0;
    for (uint32_t k = 0; k < N; k++)
        if (r.orig[k] != kNone) most += n.nfi[r.orig[k]] + n.nfo[r.orig[k]];
    r.edges.resize(most);
    uint32_t *w = r.edges.data();
    for (uint32_t k = 0; k < N; k++) {
        r.eoff[k] = (uint64_t)(w - r.edges.data());
        const uint32_t g = r.orig[k];
        if (g == kNone) {
            r.hdr[k] = RF_KILL | (k == c0 ? 0u : (uint32_t)RF_OINV);
            continue;
        }
        const uint32_t *e = n.edges.data() + n.eoff[g], nfi = n.nfi[g], nfo = n.nfo[g];
        r.hdr[k] = n.hdr[g];
        r.nfi[k] = nfi;
        for (uint32_t q = 0; q < nfi; q++) *w++ = f.value[e[q]] < 0 ? id[e[q]] : c0 + (uint32_t)f.value[e[q]];
        if (!f.observable[g]) {
            r.hdr[k] &= ~(uint32_t)(RF_MARKF0 | RF_SENS | RF_MANY);
            continue;
        }
        // the prune and the cover follow observable fan-outs only
        for (uint32_t q = 0; q < nfo; q++)
            if (f.observable[e[nfi + q]]) {
                *w++ = id[e[nfi + q]];
                r.nfo[k]++;
            }
    }
    r.edges.resize((size_t)(w - r.edges.data()));
    r.eoff[N] = r.edges.size();
    return r;
}

#endif
