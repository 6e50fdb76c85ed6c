// pdf_plan.h -- launch plans of the forward kernels: the gate records, pieces,
// far lists and shared-memory layout of one walk over a netlist.  A circuit
// has one for every gate (plane outputs, stage calls) and, when that leaves
// gates out, one for its reduced netlist (pdf_reduce.h).
#ifndef PDF_PLAN_H
#define PDF_PLAN_H

#include <cstddef>
#include <vector>

#include "pdf.h"
#include "pdf_reduce.h"

struct PlanOpts {
    uint32_t bw = 4;         // words per column block
    uint32_t threads = 0;    // the caller's block size (0: chosen)
    int regs = 0;            // registers per thread of the forward kernel (forward_kernel_regs)
    int smem_block = 0, smem_sm = 0;  // shared memory per block (opt-in) and per SM
};

// What a launch needs besides the device arrays.
struct PlanShape {
    uint32_t n_gates = 0, n_levels = 0;
    uint32_t bw = 4, threads = 512, ring = 0, ring2 = 0, farcap = 0;
    uint32_t cap = 512, ecap = 2048, n_pieces = 0, bm_shared = 0;
    uint32_t off_ring = 0, off_rec = 0, off_edge = 0, off_fid = 0, off_bm = 0, off_pbits = 0, off_mbar = 0;
    size_t fwd_smem = 0;
    uint32_t occ = 1;    // forward CTAs per SM its registers and shared memory are sized for
    uint32_t nfo_mask = 0xFFFFFFFFu;  // fan-out count bits of w[1]; the bits above: its reach (0: not kept)
    uint32_t in_pieces = 0;  // pieces of level 0 (0 when the reach is not kept)
    uint64_t chain = 0;  // length of one CTA's walk (pieces, or gates for the lane kernel)
};

// The image of a netlist that the resident kernel keeps in shared memory: 16
// bytes per gate (header; fan-ins 0..3 as 16-bit ids, of an input its row in
// the pair planes; edge offset | last level its mark reaches << 16) and one
// more for the end of the edges, 16-bit edges (fan-ins of gates with more
// than four, then fan-outs), per level its first gate and how many of its
// gates may hold a mark after the prune, and, where they fit, the caller's ids.
struct ResidentImage {
    std::vector<unsigned char> bytes;  // empty: the netlist does not fit
    uint32_t off_edge = 0, off_lvl = 0;
    bool ids = false;  // holds the caller's ids (else read from device memory)
};
// `smem`: dynamic shared memory a CTA may have.
ResidentImage build_resident(const NetPlan &n, size_t smem);

// Shared memory and column blocks of one resident walk.
struct ResidentShape {
    uint32_t bw = 0, threads = 0, per = 0, ctas = 0, occ = 0, blocks = 0;
    uint32_t off_vt = 0, off_m = 0, off_bm = 0, off_mbar = 0;
    size_t smem = 0;
    double block_us = 0;  // modelled time of one column block
    uint32_t words = 0;   // words an SM can take at a time, over all the widths that fit
    double us = 0;        // modelled time of the walk
};
struct ResidentSizes {
    uint32_t n_gates = 0, n_levels = 0, image_bytes = 0;
    uint32_t sms = 0, regs = 0;
    size_t smem_block = 0, smem_sm = 0;
};
// rows: plane rows that it stores of every gate (0: none, lean walks; 2: codes; 3: and marks).
ResidentShape resident_shape(const ResidentSizes &z, uint64_t W, uint32_t rows = 0);
// Whether such a walk is the faster one, against the staged kernel's: of the
// same netlist (up to resident_words), and (with rows, `gates` and `pieces` of
// the whole netlist) of all gates.
constexpr uint32_t kResidentWords = 8;  // words an SM has room for from which it always is
uint64_t resident_words(const ResidentShape &s, uint32_t sms);
bool resident_pays(const ResidentShape &s, uint64_t W, uint32_t sms);
bool resident_planes_pay(const ResidentShape &s, uint64_t W, uint32_t rows, uint64_t gates, uint32_t pieces);

struct LaunchPlan : PlanShape {
    std::vector<GateRec> recs;
    std::vector<Piece> pieces;
    std::vector<uint32_t> far_ids;
};

// Records only (what the cover reads), for a netlist that the resident kernel walks.
void build_records(const NetPlan &n, LaunchPlan &pl);
pdf_status build_plan(const NetPlan &n, const PlanOpts &o, LaunchPlan &pl);

#endif
