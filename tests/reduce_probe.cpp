// The host-side netlist reduction of pdf_reduce.h behind two C calls, for
// tests/test_reduced.py (compiled there with g++; no CUDA).
#include "pdf_reduce.h"

static NetPlan g_full, g_red;
static NetFacts g_facts;

extern "C" uint32_t probe_reduce(const pdf_netlist *nl, int fixed, int8_t *value, uint8_t *observable,
                                 uint8_t *needed) {
    g_full = net_plan(nl, fixed != 0);
    g_facts = net_facts(g_full, fixed != 0);
    g_red = reduce_net(g_full, g_facts);
    std::copy(g_facts.value.begin(), g_facts.value.end(), value);
    std::copy(g_facts.observable.begin(), g_facts.observable.end(), observable);
    std::copy(g_facts.needed.begin(), g_facts.needed.end(), needed);
    return g_red.n_gates();
}

// Of the netlist reduced last: arrays of [gates], level_off of [levels + 1].
extern "C" uint32_t probe_arrays(uint32_t *orig, uint32_t *hdr, uint32_t *nfi, uint32_t *nfo, uint64_t *eoff,
                                 uint32_t *edges, uint32_t *level_off) {
    std::copy(g_red.orig.begin(), g_red.orig.end(), orig);
    std::copy(g_red.hdr.begin(), g_red.hdr.end(), hdr);
    std::copy(g_red.nfi.begin(), g_red.nfi.end(), nfi);
    std::copy(g_red.nfo.begin(), g_red.nfo.end(), nfo);
    std::copy(g_red.eoff.begin(), g_red.eoff.end(), eoff);
    std::copy(g_red.edges.begin(), g_red.edges.end(), edges);
    std::copy(g_red.level_off.begin(), g_red.level_off.end(), level_off);
    return g_red.n_levels();
}
