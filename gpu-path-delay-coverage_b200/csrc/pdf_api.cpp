// pdf_api.cpp -- the C ABI (include/pdf.h) over the sm_100a kernels.
//
// Every call returns a status and never exits: the reference's HANDLE_ERROR
// exit(EXIT_FAILURE) (simkernel.cuh:32-39, markkernel.cuh:13-20,
// mergekernel.cuh:17-24, coverkernel.cuh:15-25) becomes PDF_ECUDA / PDF_EINVAL.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <future>
#include <initializer_list>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <type_traits>
#include <vector>

#include "pdf.h"
#include "pdf_inject.h"
#include "pdf_internal.h"
#include "pdf_kernels.cuh"
#include "pdf_plan.h"

#include <atomic>

namespace {
std::atomic<uint32_t> g_inject[3];
}  // namespace

bool inject_fail(int site) {
    if (site < 1 || site > 2) return false;
    uint32_t n = g_inject[site].load();
    while (n > 0)
        if (g_inject[site].compare_exchange_weak(n, n - 1)) return true;
    return false;
}
cudaError_t dev_alloc(void **p, size_t bytes) {
    if (inject_fail(PDF_INJECT_DEVICE_ALLOC)) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaMalloc(p, bytes);
}
cudaError_t host_alloc(void **p, size_t bytes) {
    if (inject_fail(PDF_INJECT_HOST_ALLOC)) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaHostAlloc(p, bytes, cudaHostAllocDefault);
}

extern "C" pdf_status pdf_test_inject(int site, uint32_t count) {
    if (site < 1 || site > 2) return PDF_EINVAL;
    g_inject[site].store(count);
    return PDF_OK;
}

namespace {


// The last failing CUDA call of this thread, for pdf_last_error().
thread_local char g_last_error[256];
static void note_cuda_error(cudaError_t e, const char *call, int line) {
    std::snprintf(g_last_error, sizeof g_last_error, "%s (%d) at pdf_api.cpp:%d: %.160s", cudaGetErrorName(e),
                  (int)e, line, call);
}

#define PDF_CUDA(call)                                  \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) {                        \
            note_cuda_error(e_, #call, __LINE__);       \
            (void)cudaGetLastError();                   \
            return e_ == cudaErrorMemoryAllocation ? PDF_ENOMEM : PDF_ECUDA; \
        }                                               \
    } while (0)

pdf_status err_status(unsigned int err) {
    if (err & kErrHashFull) return PDF_ENOMEM;
    if (err & kErrTimeout) return PDF_ETIMEOUT;
    return PDF_OK;
}

void set_msg(char *msg, size_t len, const char *fmt, unsigned long long a = 0,
             unsigned long long b = 0) {
    if (msg && len) std::snprintf(msg, len, fmt, a, b);
}

// Who else has a device block's address: batches bound to it (each binding has
// a token, dropped when the batch is bound anew or destroyed) and graphs that
// the caller captured (until the block's owner is destroyed).
struct Holders {
    std::vector<std::weak_ptr<const void>> batches;
    bool graph = false;
    bool any() const {
        for (const auto &b : batches)
            if (!b.expired()) return true;
        return graph;
    }
    void add(const std::weak_ptr<const void> &batch) {
        batches.erase(std::remove_if(batches.begin(), batches.end(), [](const auto &b) { return b.expired(); }),
                      batches.end());
        batches.push_back(batch);
    }
};

using KeptBlocks = std::vector<std::pair<void *, Holders>>;

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    Holders holders;
    void release() {
        if (p && cudaFree(p) != cudaSuccess) (void)cudaGetLastError();
        p = nullptr;
        bytes = 0;
        holders = Holders{};
    }
    // Grow to at least `need` bytes (contents are not kept).  A block that a
    // batch or a graph holds goes to `kept` instead of being freed.
    cudaError_t ensure(size_t need, KeptBlocks *kept = nullptr) {
        if (bytes >= need) return cudaSuccess;
        if (kept && p && holders.any()) {
            try {
                kept->emplace_back(p, holders);
            } catch (const std::bad_alloc &) {
                return cudaErrorMemoryAllocation;
            }
            p = nullptr;
        }
        release();
        cudaError_t e = dev_alloc(&p, need ? need : 16);
        if (e == cudaSuccess) bytes = need;
        return e;
    }
    template <class T>
    T *as() const { return static_cast<T *>(p); }
};

// Scoped device selection.
struct DeviceGuard {
    int prev = -1;
    bool ok = false;
    // Every entry point that touches the device starts here.  Its launches
    // are checked with cudaGetLastError, which would also report a failure
    // that an earlier call on this thread left unchecked (the caller's own,
    // say), so that slot is cleared first; errors that poison the context
    // come back from every later call anyway.  A failure here is reported
    // through `ok` and not left pending for the caller's next check.
    explicit DeviceGuard(int dev) {
        (void)cudaGetLastError();
        if (cudaGetDevice(&prev) != cudaSuccess) {
            prev = -1;
            (void)cudaGetLastError();
        }
        ok = cudaSetDevice(dev) == cudaSuccess;
        if (!ok) (void)cudaGetLastError();
    }
    ~DeviceGuard() {
        if (prev >= 0 && cudaSetDevice(prev) != cudaSuccess) (void)cudaGetLastError();
    }
};

}  // namespace

// Per-batch device workspace (owned by a state, or by a circuit for the
// stage calls).
struct Workspace {
    DevBuf scratch;            // one block, laid out by scratch_of
    WideSync *sync = nullptr;  // wide kernel: its barrier counters, zero between launches (in the owner's block)
    DevBuf pi_counts;          // pdf_cover_counts: paths per (primary input, pair)
    DevBuf seg_first;          // (net, pair) hash set of the cover with segments
    uint64_t seg_first_mask = 0;
    DevBuf planes;  // internal V, T, M planes when the caller gives none
    DevBuf pi;      // staged host pairs
    // blocks that were outgrown while held: calls of one walk (with planes, say)
    // grow a state's workspace past what a batch of the other was bound to
    KeptBlocks kept;
    // From here on the current blocks belong to a graph that the caller
    // captures, or also to the binding of a batch; false: out of host memory.
    void hold_for_graph() { scratch.holders.graph = seg_first.holders.graph = planes.holders.graph = pi.holders.graph = true; }
    bool hold_for(const std::weak_ptr<const void> &batch) {
        try {
            for (DevBuf *b : {&scratch, &seg_first, &planes, &pi}) b->holders.add(batch);
        } catch (const std::bad_alloc &) {
            return false;
        }
        return true;
    }
    // frees the kept blocks that nobody holds any more
    void sweep() {
        const auto gone = std::remove_if(kept.begin(), kept.end(), [](const auto &k) {
            if (k.second.any()) return false;
            if (cudaFree(k.first) != cudaSuccess) (void)cudaGetLastError();
            return true;
        });
        kept.erase(gone, kept.end());
    }
    void release() {
        scratch.release();
        pi_counts.release();
        seg_first.release();
        seg_first_mask = 0;
        planes.release();
        pi.release();
        for (const auto &k : kept)
            if (cudaFree(k.first) != cudaSuccess) (void)cudaGetLastError();
        kept.clear();
    }
};

namespace {

// One walk over a netlist, on the device.
struct Plan : PlanShape {
    DevCircuit dc{};
    const Piece *pieces = nullptr;
    const uint32_t *far_ids = nullptr;
    bool wide = false;  // its staged walk is the wide kernel's (a lane plan)
    uint32_t mean_width = 0;
    // the resident kernel's image of the netlist (null: it does not fit)
    const void *image = nullptr;
    uint32_t off_edge_im = 0, off_lvl_im = 0, image_ids = 0;
    ResidentSizes res;
    void bind(const LaunchPlan &l, const NetPlan &n, const ResidentImage &im, const unsigned char *base,
              const struct PlanOffsets &o);
};

// One call's walk over W words of pairs: the plan, the kernel and its column
// block.
struct Walk {
    const Plan *p = nullptr;
    uint32_t bw = 0;
    bool resident = false;
    int out = RES_LEAN;  // resident: the planes it writes
    // wide kernel: words per lane (0: not it), its chunks per segment and segments
    uint32_t wide = 0, cps = 0, nseg = 0, chunks = 0;
    // the cover's bitmaps are per kLaneCoverWords words
    bool fine() const { return wide || (!resident && lane_tile(bw)); }
    ResidentShape rs;
};

struct PlanOffsets {
    size_t rec = 0, edges = 0, level_off = 0, pieces = 0, far = 0, orig = 0, image = 0;
};

void Plan::bind(const LaunchPlan &l, const NetPlan &n, const ResidentImage &im, const unsigned char *base,
                const PlanOffsets &o) {
    static_cast<PlanShape &>(*this) = l;
    dc.rec = reinterpret_cast<const GateRec *>(base + o.rec);
    dc.edges = reinterpret_cast<const uint32_t *>(base + o.edges);
    dc.level_off = reinterpret_cast<const uint32_t *>(base + o.level_off);
    dc.orig = n.orig.empty() ? nullptr : reinterpret_cast<const uint32_t *>(base + o.orig);
    dc.n_gates = n_gates;
    dc.n_levels = n_levels;
    dc.nfo_mask = nfo_mask;
    pieces = reinterpret_cast<const Piece *>(base + o.pieces);
    far_ids = reinterpret_cast<const uint32_t *>(base + o.far);
    if (im.bytes.empty()) return;
    image = base + o.image;
    off_edge_im = im.off_edge;
    off_lvl_im = im.off_lvl;
    image_ids = im.ids ? 1u : 0u;
    res.n_gates = n_gates;
    res.n_levels = n_levels;
    res.image_bytes = (uint32_t)im.bytes.size();
}

// Arrays of a circuit on their way into one device block: small circuits go
// in one copy through a host image, large ones array by array.
struct PlanUpload {
    struct Part {
        const void *src;
        size_t off, bytes;
    };
    std::vector<Part> parts;
    size_t bytes = 0;
    size_t add(const void *src, size_t n) {
        const size_t off = bytes;
        parts.push_back({src, off, n});
        bytes = (off + n + 255) & ~(size_t)255;
        return off;
    }
    PlanOffsets add_plan(const NetPlan &n, const LaunchPlan &l, const ResidentImage &im) {
        PlanOffsets o;
        o.rec = add(l.recs.data(), l.recs.size() * sizeof(GateRec));
        o.edges = add(n.edges.data(), n.edges.size() * 4);
        bytes += 256;  // bulk copies of edge slices are rounded up to 16 bytes
        o.level_off = add(n.level_off.data(), n.level_off.size() * 4);
        o.pieces = add(l.pieces.data(), l.pieces.size() * sizeof(Piece));
        o.far = add(l.far_ids.data(), l.far_ids.size() * 4);
        o.orig = add(n.orig.data(), n.orig.size() * 4);
        o.image = add(im.bytes.data(), im.bytes.size());
        return o;
    }
    // Done when it returns: work on streams that do not wait for the legacy
    // stream may follow at once.
    bool copy(unsigned char *dst) const { return put(dst) && cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess; }
    bool put(unsigned char *dst) const {
        if (bytes <= (1u << 20)) {
            std::vector<unsigned char> img(bytes, 0);
            for (const Part &p : parts)
                if (p.src && p.bytes) std::memcpy(img.data() + p.off, p.src, p.bytes);
            return cudaMemcpy(dst, img.data(), bytes, cudaMemcpyHostToDevice) == cudaSuccess;
        }
        for (const Part &p : parts) {
            if (!p.bytes) continue;
            const cudaError_t e = p.src ? cudaMemcpy(dst + p.off, p.src, p.bytes, cudaMemcpyHostToDevice)
                                        : cudaMemset(dst + p.off, 0, p.bytes);
            if (e != cudaSuccess) return false;
        }
        return true;
    }
};

}  // namespace

struct pdf_circuit {
    int device = 0;
    int mark_mode = PDF_MARK_DEFAULT;
    pdf_circuit_info info{};
    DevBuf mem;  // both plans' arrays and stage.sync
    // the stage calls' error word: mapped host memory, from the first such call
    // on (read after the call's sync, without a copy)
    uint32_t *host_err = nullptr, *err = nullptr;
    uint32_t bw = 4;  // the tile: column block of the full walk, divisor of the device planes' pitch
    Plan full, red;   // every gate; the reduced netlist (n_gates 0: none)
    // the plan of grading calls that ask for no plane
    const Plan &lean() const { return red.n_gates ? red : full; }
    // Plans at the tile for the staged kernels, of the reduced netlist and of all
    // gates, built when first asked for: of circuits whose single calls take
    // another column block (narrower ones, single_tile; the wide kernel's) or
    // walk a reduced netlist on chip.
    struct TilePlan {
        bool wanted = false;
        PlanOpts opts;
        NetPlan net;
        DevBuf mem;
        Plan plan;
        std::mutex mu;
    };
    mutable TilePlan tile_red, tile_full;
    uint64_t narrow_words = ~0ull;  // single calls over more words than this take them
    const Plan &at_tile(TilePlan &t, const Plan &otherwise) const;
    // The lean calls' plan for the staged kernels, at the tile; of a reduced
    // netlist that fits on chip, null where it could not be built.
    const Plan *lean_at_tile() const {
        const Plan &p = red.n_gates ? at_tile(tile_red, red) : at_tile(tile_full, full);
        return &p == &red && red.image ? nullptr : &p;
    }
    // Planes from the resident kernel: every gate whose value is not constant,
    // where they fit on chip (the constant rows are filled in), else null.
    Plan live;
    const Plan *out_plan = nullptr;
    const int8_t *value = nullptr;  // [n_gates] the constant value, or -1
    // The wide kernel's shape with lw words per lane: the segment length with
    // the fewest rounds of chunks (and about 1.5 chunks' worth per gate).
    void wide_shape(Walk &k, uint64_t W, uint32_t lw) const {
        k.wide = lw;
        k.chunks = (uint32_t)((W + 32 * lw - 1) / (32 * lw));
        const uint64_t warps = (uint64_t)k.p->res.sms * kWideCtas * (kWideThreads / 32);
        double best = 0;
        for (uint32_t cps = 1; cps <= 8; cps *= 2) {
            const uint64_t items = (uint64_t)k.p->mean_width * ((k.chunks + cps - 1) / cps);
            const double t = (double)((items + warps - 1) / warps) * (cps + 1.5);
            if (!k.cps || t < best) {
                k.cps = cps;
                best = t;
            }
        }
        k.nseg = (k.chunks + k.cps - 1) / k.cps;
    }
    // the staged kernels' walk of plan p over W words
    Walk staged_walk(const Plan &p, uint64_t W) const {
        Walk k;
        k.p = &p;
        k.bw = p.bw;
        if (p.wide) wide_shape(k, W, 2);
        return k;
    }
    Walk full_walk(uint64_t W) const { return staged_walk(W > narrow_words ? at_tile(tile_full, full) : full, W); }
    Walk lean_walk(uint64_t W) const {
        if (lean().image) {
            const Walk k = resident_walk(lean(), W, RES_LEAN);
            if (resident_pays(k.rs, W, lean().res.sms)) return k;
            const Plan *p = red.n_gates || W > narrow_words ? lean_at_tile() : &full;
            return p ? staged_walk(*p, W) : k;
        }
        return staged_walk(W > narrow_words ? *lean_at_tile() : lean(), W);
    }
    // A batch's: its circuits share the GPU, so a wide plan takes the lane kernel
    // (lanes) or the plan at the tile, and a netlist that fits on chip may be
    // walked there (chip) or not.
    Walk batch_walk(uint64_t W, bool lanes, bool chip) const {
        Walk k;
        const bool on_chip = lean().image && chip;
        if (!on_chip) k.p = lean().wide && lanes ? &lean() : lean_at_tile();
        if (!k.p) return resident_walk(lean(), W, RES_LEAN);
        k.bw = k.p->bw;
        return k;
    }
    static Walk resident_walk(const Plan &p, uint64_t W, int out) {
        Walk k;
        k.p = &p;
        k.resident = true;
        k.out = out;
        k.rs = resident_shape(p.res, W, out == RES_LEAN ? 0 : out == RES_SIM ? 2 : 3);
        k.bw = k.rs.bw;
        return k;
    }
    // the walk of calls that ask for planes: all three, or the codes alone (out = RES_SIM)
    Walk planes_walk(uint64_t W, int out = RES_PLANES) const {
        if (out_plan) {
            const Walk k = resident_walk(*out_plan, W, out);
            if (resident_planes_pay(k.rs, W, out == RES_SIM ? 2 : 3, info.n_gates, full.n_pieces)) return k;
        }
        return full_walk(W);
    }
    uint32_t hash_cap = 4096, cover_threads = 256, cover_grid = 0;
    uint32_t small_cap = 0;  // nets per pair of the cover's small-table pass
    uint32_t wait_polls = 0;  // bound of the forward kernels' waits (0 = the default)
    Workspace stage;  // scratch of the stage calls
    std::mutex mu;    // serialises the stage scratch
    // segments longer than one net
    uint32_t seg_len = 1;
    uint64_t n_segs = 0;
    DevBuf segs, seg_off;
    // entries of a state's first-detect arrays: one per segment
    uint64_t n_first() const { return seg_len > 1 ? n_segs : info.n_gates; }
    SegArgs seg_args() const {
        SegArgs a{};
        if (seg_len > 1) {
            a.segs = segs.as<uint32_t>();
            a.seg_off = seg_off.as<uint32_t>();
            a.N = seg_len;
            a.S = (uint32_t)n_segs;
        }
        return a;
    }
};

struct ProfEvents {
    cudaEvent_t ev[4];  // call start, forward end, cover end, call end
};

struct pdf_state {
    pdf_circuit *c = nullptr;
    int device = 0;  // the circuit's device (destroy does not need the circuit)
    DevBuf mem;  // first-detect ids, falling then rising, the accumulators, ws.sync
    struct Ref {
        void *p = nullptr;
        template <class T>
        T *as() const { return static_cast<T *>(p); }
    } first_x, first_y, acc;
    // two host copies of the accumulators (pinned and mapped): [0] read back by
    // DMA after a stream sync, [1] the mirror, which whatever changes the totals
    // writes too: the cover kernel that closes a batch, a reset, a restore
    DevAcc *host_acc = nullptr;
    DevAcc *mirror = nullptr;  // device address of host_acc[1]
    Workspace ws;
    std::mutex mu;
    bool profiling = false;
    std::vector<ProfEvents> prof;   // one entry per profiled call
    std::vector<ProfEvents> pool;   // recycled events
    ProfEvents *pe = nullptr;       // events of the call in progress
    // the batch marked by pdf_grade_mark_async and not yet counted
    bool pending = false;
    Walk pend_walk;
    const uint32_t *pend_M = nullptr;
    uint64_t pend_ld = 0, pend_n = 0, pend_base = 0;
};

namespace {
void prof_release(std::vector<ProfEvents> &v) {
    for (auto &p : v)
        for (auto &e : p.ev) cudaEventDestroy(e);
    v.clear();
}
}  // namespace

// ---------------------------------------------------------------------------

extern "C" const char *pdf_last_error(void) { return g_last_error; }

extern "C" const char *pdf_status_string(int s) {
    switch (s) {
        case PDF_OK: return "ok";
        case PDF_EINVAL: return "invalid argument";
        case PDF_ENOMEM: return "out of memory";
        case PDF_EOVERFLOW: return "path count overflow";
        case PDF_ETIMEOUT: return "device wait timed out";
        case PDF_ECUDA: return "CUDA error";
        case PDF_ENOTSUP: return "not supported";
        case PDF_EBUSY: return "busy";
        case PDF_ENODEV: return "no CUDA device";
        case PDF_ELIMIT: return "request exceeds the fixed scratch of an allocation-free call";
        default: return "unknown status";
    }
}

extern "C" int pdf_abi_version(void) { return PDF_ABI_VERSION; }

extern "C" pdf_status pdf_netlist_check(const pdf_netlist *nl, char *msg, size_t len) {
    if (!nl) {
        set_msg(msg, len, "null netlist");
        return PDF_EINVAL;
    }
    const uint32_t G = nl->n_gates, L = nl->n_levels;
    if (G == 0 || G == 0xFFFFFFFFu || L == 0 || !nl->level_offsets || !nl->type || !nl->po ||
        !nl->nfi || !nl->nfo || !nl->edge_offset || (!nl->edges && nl->n_edges)) {
        set_msg(msg, len, "empty netlist or missing array");
        return PDF_EINVAL;
    }
    if (nl->n_edges >= 0xFFFFFFFFull) {
        set_msg(msg, len, "too many edges (%llu)", nl->n_edges);
        return PDF_EINVAL;
    }
    if (nl->level_offsets[0] != 0 || nl->level_offsets[L] != G) {
        set_msg(msg, len, "level_offsets must start at 0 and end at n_gates");
        return PDF_EINVAL;
    }
    for (uint32_t l = 0; l < L; l++)
        if (nl->level_offsets[l + 1] < nl->level_offsets[l]) {
            set_msg(msg, len, "level_offsets decrease at level %llu", l);
            return PDF_EINVAL;
        }
    const uint32_t npi = nl->level_offsets[1];
    if (npi == 0) {
        set_msg(msg, len, "level 0 (primary inputs) is empty");
        return PDF_EINVAL;
    }
    // A gate's fan-ins lie below its level's first gate, its fan-outs at or
    // past the next level's.  Fan-in uses are counted on the way.
    std::vector<uint32_t> start((size_t)G + 1, 0);  // [g + 1]: fan-in uses of g
    uint64_t uses = 0;
    for (uint32_t l = 0; l < L; l++) {
        const uint32_t lo = nl->level_offsets[l], hi = nl->level_offsets[l + 1];
        for (uint32_t g = lo; g < hi; g++) {
            const uint32_t t = nl->type[g], nfi = nl->nfi[g], nfo = nl->nfo[g];
            if (t >= PDF_NTYPES) {
                set_msg(msg, len, "gate %llu: unknown type code %llu", g, t);
                return PDF_EINVAL;
            }
            if (nl->po[g] > 1) {
                set_msg(msg, len, "gate %llu: po must be 0 or 1", g);
                return PDF_EINVAL;
            }
            if ((t == PDF_INPT) != (g < npi)) {
                set_msg(msg, len, "gate %llu: INPT gates must be exactly level 0", g);
                return PDF_EINVAL;
            }
            if (t == PDF_INPT ? nfi != 0 : (nfi == 0 || nfi > 255)) {
                set_msg(msg, len, "gate %llu: bad fan-in count %llu", g, nfi);
                return PDF_EINVAL;
            }
            const uint64_t end = nl->edge_offset[g] + (uint64_t)nfi + nfo;
            if (end > nl->n_edges || end < nl->edge_offset[g]) {
                set_msg(msg, len, "gate %llu: edge range out of bounds", g);
                return PDF_EINVAL;
            }
            if ((uses += (uint64_t)nfi + nfo) >= 0xFFFFFFFFull) {  // lists that overlap can add up to more than n_edges
                set_msg(msg, len, "too many edges (%llu)", uses);
                return PDF_EINVAL;
            }
            const uint32_t *e = nl->edges + nl->edge_offset[g];
            for (uint32_t j = 0; j < nfi; j++) {
                if (e[j] >= lo) {
                    set_msg(msg, len, "gate %llu: fan-in %llu not on a lower level", g, e[j]);
                    return PDF_EINVAL;
                }
                start[e[j] + 1]++;
            }
            for (uint32_t k = 0; k < nfo; k++) {
                const uint32_t f = e[nfi + k];
                if (f >= G || f < hi) {
                    set_msg(msg, len, "gate %llu: fan-out %llu not on a higher level", g, f);
                    return PDF_EINVAL;
                }
            }
        }
    }
    // Fan-out lists must be the transpose of the fan-in lists (as multisets).
    for (uint32_t g = 0; g < G; g++)
        if (start[g + 1] != nl->nfo[g]) {
            set_msg(msg, len, "gate %llu: fan-out count %llu differs from its fan-in uses", g,
                    nl->nfo[g]);
            return PDF_EINVAL;
        }
    // Multiset comparison: the consumers of each gate (transposed from the
    // fan-in lists by a counting sort, hence ascending) against its fan-out
    // list, sorted when it does not ascend already.
    for (uint32_t g = 0; g < G; g++) start[g + 1] += start[g];
    std::vector<uint32_t> cons(start[G]), fill(start.begin(), start.end() - 1), fo;
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t *e = nl->edges + nl->edge_offset[g];
        for (uint32_t j = 0; j < nl->nfi[g]; j++) cons[fill[e[j]]++] = g;
    }
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t *e = nl->edges + nl->edge_offset[g] + nl->nfi[g], *want = cons.data() + start[g];
        if (std::equal(e, e + nl->nfo[g], want)) continue;
        fo.assign(e, e + nl->nfo[g]);
        std::sort(fo.begin(), fo.end());
        if (!std::equal(fo.begin(), fo.end(), want)) {
            set_msg(msg, len, "fan-out lists are not the transpose of the fan-in lists (gate %llu)", g);
            return PDF_EINVAL;
        }
    }
    set_msg(msg, len, "ok");
    return PDF_OK;
}

// ---------------------------------------------------------------------------

namespace {

// Segments of N nets (2..8): every directed subpath of N nets, listed by
// first net ascending, then depth first along fan-outs in edge order (the
// reference's generateSegmentList lives in its missing util/segment.cuh).
// Counted first (paths of k nets from g = sum over fan-outs of paths of k - 1
// nets), then written as [S][N] with a CSR offset per first net.
constexpr uint64_t kMaxSegWords = 1ull << 28;  // S * N gate ids at most (1 GiB)

pdf_status build_segments(pdf_circuit *c, const pdf_netlist *nl, uint32_t N) {
    const uint32_t G = nl->n_gates;
    auto fo = [&](uint32_t g, uint32_t k) { return nl->edges[nl->edge_offset[g] + nl->nfi[g] + k]; };
    std::vector<uint64_t> cnt(G, 1), nxt(G);
    for (uint32_t k = 1; k < N; k++) {
        for (uint32_t g = 0; g < G; g++) {
            uint64_t t = 0;
            for (uint32_t j = 0; j < nl->nfo[g]; j++) t = std::min(t + cnt[fo(g, j)], kMaxSegWords + 1);
            nxt[g] = t;
        }
        cnt.swap(nxt);
    }
    std::vector<uint32_t> off(G + 1, 0);
    uint64_t S = 0;
    for (uint32_t g = 0; g < G; g++) {
        S += cnt[g];
        if (S * N > kMaxSegWords) return PDF_ENOTSUP;
        off[g + 1] = (uint32_t)S;
    }
    std::vector<uint32_t> segs;
    try {
        segs.resize(S * N);
    } catch (const std::bad_alloc &) {
        return PDF_ENOMEM;
    }
    uint32_t path[8], idx[8];
    uint64_t w = 0;
    for (uint32_t g0 = 0; g0 < G; g0++) {
        int d = 0;
        path[0] = g0;
        idx[0] = 0;
        while (d >= 0) {
            if ((uint32_t)d == N - 1) {
                std::memcpy(segs.data() + w, path, N * 4);
                w += N;
                d--;
            } else if (idx[d] < nl->nfo[path[d]]) {
                path[d + 1] = fo(path[d], idx[d]++);
                idx[d + 1] = 0;
                d++;
            } else {
                d--;
            }
        }
    }
    if (w != S * N) return PDF_EINVAL;
    if (c->segs.ensure(std::max<uint64_t>(S * N * 4, 16)) != cudaSuccess ||
        c->seg_off.ensure((uint64_t)(G + 1) * 4) != cudaSuccess)
        return PDF_ENOMEM;
    if ((S && cudaMemcpy(c->segs.p, segs.data(), S * N * 4, cudaMemcpyHostToDevice) != cudaSuccess) ||
        cudaMemcpy(c->seg_off.p, off.data(), (uint64_t)(G + 1) * 4, cudaMemcpyHostToDevice) != cudaSuccess)
        return PDF_ECUDA;
    c->seg_len = N;
    c->n_segs = S;
    return PDF_OK;
}

}  // namespace

namespace {

// Levels wide enough for the wide kernel: its rounds then outweigh its grid
// barriers (about 2 us a level).  Kernel times (us) at the thread-per-gate
// kernel and at this one: 3,550 gates a level and 32,768 pairs with planes
// 4,032 and 1,200; 1,500 a level and 65,536 pairs without 1,733 and 895; 308
// a level and 32,768 pairs with planes 277 and 445.  Whole calls with planes
// near the line: 1,108 gates a level (20 levels), 32 pairs 416 and 239, 65,536
// pairs 1,517 and 753; 1,038 a level (40 levels) 545 and 291, 2,141 and 1,036.
constexpr uint64_t kWideLevel = 1024;

// Column block of single calls over at most `words` words when the caller asked
// for no tile: the narrowest of 1, 2 and 4 words with at most one CTA per SM.
// A walk is a chain of levels, whose steps are shorter with fewer words.
// Measured (us; blocks of 1, 2, 4 words), four stage calls over 20,000 gates
// without XOR: 96 words 329, 349, 388; 256 words 398, 348, 387; 384 words 660,
// 432, 403; 45,000 gates FIXED: 96 words 2,101, 2,270, 2,429; 256 words 3,239,
// 2,994, 3,195; 384 words 3,811, 3,649, 3,363.
uint32_t single_tile(uint32_t bw, uint64_t words, uint64_t sms) {
    if (bw != 4 || words > 2 * sms) return bw;
    return words > sms ? 2 : 1;
}

// Mean width of the levels above the inputs.
uint64_t mean_level(const NetPlan &n) {
    return n.n_levels() > 1 ? (n.n_gates() - n.level_off[1]) / (n.n_levels() - 1) : 0;
}

// Column block of the reduced walk of a circuit whose tile is bw words, by
// the mean width of its levels above the inputs.  Narrow levels leave most
// warps of the lane kernel without a gate.
uint32_t reduced_tile(uint32_t bw, uint64_t mean_width) {
    if (lane_tile(bw) && mean_width < 512) return 4;
    return bw;
}

// A batch's circuits with wide levels take the lane kernel from this many of
// its CTAs on, else the thread-per-gate kernel at the tile: a lane CTA takes a
// level's gates 32 at a time, so few of them leave the GPU waiting for one
// another's chains.  Measured (us a pass, robust table, no XOR; lane kernel at
// 32 words and thread per gate at 4): 150,000 gates, 40 levels: 4 lane CTAs
// 3,157 and 1,060, 48: 5,525 and 4,266, 64: 5,234 and 4,776, 96: 6,030 and
// 6,975, 192: 9,293 and 11,455; 60,000 gates, 30 levels: 4: 1,510 and 464, 64:
// 2,299 and 1,935, 96: 2,616 and 2,819; FIXED 4: 3,272 and 1,571, 64: 11,100 and
// 10,619, 96: 14,994 and 15,349.
uint64_t batch_lanes_from(uint64_t sms) { return sms * 9 / 16; }

}  // namespace

// Where it cannot be built (out of memory, too many pieces) the call walks the
// plan there is, and the next one tries again.
const Plan &pdf_circuit::at_tile(TilePlan &t, const Plan &otherwise) const {
    if (!t.wanted) return otherwise;
    std::lock_guard<std::mutex> lk(t.mu);
    if (t.plan.n_gates) return t.plan;
    try {
        PlanOpts po = t.opts;
        po.regs = forward_kernel_regs((int)po.bw, mark_mode);
        LaunchPlan l;
        if (build_plan(t.net, po, l) != PDF_OK) return otherwise;
        PlanUpload up;
        const PlanOffsets at = up.add_plan(t.net, l, ResidentImage{});
        if (t.mem.ensure(up.bytes) != cudaSuccess || !up.copy(t.mem.as<unsigned char>())) {
            (void)cudaGetLastError();
            return otherwise;
        }
        t.plan.bind(l, t.net, ResidentImage{}, t.mem.as<unsigned char>(), at);
        t.net = NetPlan{};
    } catch (const std::bad_alloc &) {
        return otherwise;
    }
    return t.plan;
}

extern "C" pdf_status pdf_circuit_create(const pdf_netlist *nl, const pdf_circuit_opts *opts,
                                         pdf_circuit **out) {
    if (!out) return PDF_EINVAL;
    *out = nullptr;
    pdf_status st = pdf_netlist_check(nl, nullptr, 0);
    if (st != PDF_OK) return st;
    pdf_circuit_opts o{};
    if (opts) o = *opts;
    if (o.mark_mode < PDF_MARK_DEFAULT || o.mark_mode > PDF_MARK_FIXED_NONROBUST) return PDF_EINVAL;
    if (o.seg_len > 8) return PDF_EINVAL;
    if (o.tile_words && o.tile_words != 1 && o.tile_words != 2 && o.tile_words != 4 && o.tile_words != 8 &&
        !lane_tile(o.tile_words))
        return PDF_EINVAL;
    if (o.threads && (o.threads < 64 || o.threads > 1024 || o.threads % 32)) return PDF_EINVAL;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        (void)cudaGetLastError();
        return PDF_ENODEV;
    }
    if (o.device < 0 || o.device >= ndev) return PDF_EINVAL;
    DeviceGuard dg(o.device);
    if (!dg.ok) return PDF_ECUDA;

    // source words address gates with 31 bits and slots with 30 (pdf_device.cuh)
    if (nl->n_gates >= SRC_FAR) return PDF_ENOTSUP;
    pdf_circuit *c = new (std::nothrow) pdf_circuit();
    if (!c) return PDF_ENOMEM;
    c->device = o.device;
    c->mark_mode = o.mark_mode;
    c->wait_polls = o.wait_polls;
    const uint32_t G = nl->n_gates, L = nl->n_levels;
    pdf_circuit_info &inf = c->info;
    inf.n_gates = G;
    inf.n_levels = L;
    inf.n_pi = nl->level_offsets[1];
    inf.n_edges = nl->n_edges;
    for (uint32_t g = 0; g < G; g++) {
        inf.n_po += nl->po[g] ? 1 : 0;
        inf.max_nfi = std::max(inf.max_nfi, nl->nfi[g]);
        inf.max_nfo = std::max(inf.max_nfo, nl->nfo[g]);
    }
    for (uint32_t l = 0; l < L; l++)
        inf.max_level_width = std::max(inf.max_level_width, nl->level_offsets[l + 1] - nl->level_offsets[l]);

    // Launch plan: CTAs of `threads` threads own `bw` words of pairs; two
    // CTAs per SM share its shared memory.
    struct {
        int sharedMemPerBlockOptin = 0, sharedMemPerMultiprocessor = 0, multiProcessorCount = 0;
    } prop;
    if (cudaDeviceGetAttribute(&prop.sharedMemPerBlockOptin, cudaDevAttrMaxSharedMemoryPerBlockOptin, o.device) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&prop.sharedMemPerMultiprocessor, cudaDevAttrMaxSharedMemoryPerMultiprocessor,
                               o.device) != cudaSuccess ||
        cudaDeviceGetAttribute(&prop.multiProcessorCount, cudaDevAttrMultiProcessorCount, o.device) != cudaSuccess) {
        delete c;
        return PDF_ECUDA;
    }
    // Default tile.  The lane kernel (a warp per gate) when the circuit's
    // largest batch gives it at least one 1,024-pair column block per SM and
    // its levels average 1,024 gates or more; of its tiles the one with the
    // least modelled time, waves of CTAs (one per SM) x words per CTA x the
    // tile's time per word relative to 32 words, measured on a batch that
    // fills the GPU: 1.0, 0.67, 0.52 at 32, 64, 128 words.  (1M gates, 5,000-
    // gate levels, 262,144 pairs: 61, 36 and 58 ms at 32, 64, 128 words, 128
    // CTAs being one wave at 64 words and 64 CTAs leaving half the SMs idle
    // at 128.)  On narrower or smaller jobs the lane kernel's few CTAs leave
    // SMs idle (20,000 gates, 32,768 pairs: 0.92 against 0.25 ms): 4 words
    // (128 pairs) per CTA, or 8 when the largest batch still gives at least
    // two 8-word CTAs per SM, which halves the per-gate work of record decode
    // and staging per pair (1M gates: 137 ms at 8 words against 165 ms at 4).
    const uint64_t max_words = ((o.max_pairs ? o.max_pairs : 65536ull) + 31) / 32;
    const uint64_t mean_width = L > 1 ? (G - inf.n_pi) / (L - 1) : G;
    const uint64_t sms = (uint64_t)prop.multiProcessorCount;
    if (o.tile_words) {
        c->bw = o.tile_words;
    } else if (max_words / kLaneWords >= sms && mean_width >= 1024) {
        double best = 0;
        for (const auto &t : {std::make_pair(kLaneWords, 1.0), std::make_pair(kLaneWords2, 0.67),
                              std::make_pair(kLaneWords4, 0.52)}) {
            const uint64_t ctas = (max_words + t.first - 1) / t.first;
            const double cost = (double)((ctas + sms - 1) / sms) * t.first * t.second;
            if (!best || cost < best) {
                best = cost;
                c->bw = t.first;
            }
        }
    } else {
        c->bw = max_words / 8 >= 2ull * sms ? 8u : 4u;
    }
    const bool fixed = o.mark_mode >= PDF_MARK_FIXED_ROBUST;
    PlanOpts po;
    // a caller that asks for a tile gets its kernel for the whole walk (the
    // reduced one takes the wide kernel unless a thread per gate was asked for)
    const bool wide_full = !o.tile_words && mean_width >= kWideLevel;
    bool wide_red = false;
    const uint32_t wide_bw = lane_tile(c->bw) ? c->bw : kLaneWords;  // (a batch's lane kernel)
    const uint32_t single_bw = o.tile_words || wide_full ? c->bw : single_tile(c->bw, max_words, sms);
    if (single_bw != c->bw) c->narrow_words = single_bw * sms;
    po.bw = wide_full ? wide_bw : single_bw;
    po.threads = o.threads;
    po.regs = forward_kernel_regs((int)po.bw, o.mark_mode);
    po.smem_block = prop.sharedMemPerBlockOptin;
    po.smem_sm = prop.sharedMemPerMultiprocessor;
    // Canonical edge array: each gate's fan-ins then fan-outs, gates in id
    // order, so that a run of gates owns one contiguous slice (staged into
    // shared memory by a bulk copy).
    NetPlan net = net_plan(nl, fixed);
    LaunchPlan full, red;
    // The plan of the whole netlist is built on a second thread where there
    // is enough of it, beside the reduced netlist and its plan here.
    std::future<pdf_status> other;
    if (G >= 16384 && o.seg_len <= 1) {
        try {
            other = std::async(std::launch::async, [&net, po, &full] { return build_plan(net, po, full); });
        } catch (const std::system_error &) {  // no thread to be had
        }
    }
    pdf_status pst = PDF_OK;
    if (!other.valid()) pst = build_plan(net, po, full);
    // The reduced netlist (single nets only: a circuit with segments walks every
    // gate), and the resident kernel's image of what a lean call walks.
    NetPlan rnet, lnet;
    ResidentImage image, limage;
    LaunchPlan live;
    std::vector<int8_t> value;
    enum { kNoOut, kOutFull, kOutRed, kOutLive } out_of = kNoOut;  // whose image writes planes
    const size_t res_smem = (size_t)prop.sharedMemPerBlockOptin - 1024;
    if (pst == PDF_OK && o.seg_len <= 1) {
        NetFacts facts = net_facts(net, fixed);
        const bool reduced = facts.n_needed <= (uint64_t)G * 9 / 10;
        if (reduced) rnet = reduce_net(net, facts);
        image = build_resident(reduced ? rnet : net, res_smem - 1024);
        if (reduced && !image.bytes.empty()) {
            build_records(rnet, red);
            c->tile_red.wanted = true;
            c->tile_red.opts.bw = reduced_tile(c->bw, mean_level(rnet));
        } else if (reduced) {
            PlanOpts ro = po;
            const uint64_t rw = mean_level(rnet);
            wide_red = (!o.tile_words || lane_tile(o.tile_words)) && rw >= kWideLevel;
            const uint32_t tile = reduced_tile(c->bw, rw);
            ro.bw = wide_red ? wide_bw : single_bw != c->bw ? single_bw : tile;
            ro.threads = wide_red ? 0 : o.threads;
            if (ro.bw != po.bw) ro.regs = forward_kernel_regs((int)ro.bw, o.mark_mode);
            pst = build_plan(rnet, ro, red);
            c->tile_red.wanted = ro.bw != tile;
            c->tile_red.opts.bw = tile;
            // no plan of the reduced netlist (the thread-per-gate kernel takes
            // 65,536 pieces at most, the lane kernel any number): lean calls
            // walk all of it
            if (pst == PDF_ENOTSUP) {
                rnet = NetPlan{};
                red = LaunchPlan{};
                wide_red = c->tile_red.wanted = false;
                pst = PDF_OK;
            }
        }
        // planes: what the lean image holds if that is all that is not
        // constant, else an image of its own
        uint64_t n_live = 0;
        for (uint32_t g = 0; g < G; g++) n_live += facts.value[g] < 0;
        if (!image.bytes.empty() && !reduced) {
            out_of = kOutFull;
        } else if (!image.bytes.empty() && n_live == facts.n_needed) {
            out_of = kOutRed;
        } else if (n_live * 28 <= res_smem) {
            for (uint32_t g = 0; g < G; g++) facts.needed[g] = facts.value[g] < 0;
            facts.n_needed = n_live;
            lnet = reduce_net(net, facts);
            limage = build_resident(lnet, res_smem - 1024);
            if (!limage.bytes.empty()) {
                build_records(lnet, live);
                out_of = kOutLive;
            }
        }
        if (out_of == kOutFull) value.assign(G, -1);  // its walk writes every row
        else if (out_of != kNoOut) value.swap(facts.value);
    }
    if (other.valid()) {
        const pdf_status fst = other.get();
        if (fst != PDF_OK) pst = fst;
    }
    // (a wide plan of all gates is walked by batches only where it is the lean one)
    c->tile_full.wanted =
        po.bw != c->bw && (!wide_full || (o.seg_len <= 1 && !rnet.n_gates()));
    c->tile_full.opts.bw = c->bw;
    if (pst != PDF_OK) {
        delete c;
        return pst;
    }
    // nets one pair may mark in the cover: as many as its shared memory holds
    c->hash_cap = 4096;
    while (c->hash_cap > 256 && cover_smem_bytes(c->hash_cap) > (size_t)prop.sharedMemPerBlockOptin) c->hash_cap -= 256;
    c->small_cap = std::min(cover_small_cap(o.device, nullptr), c->hash_cap);
    if (c->small_cap < 256) {  // (the level table comes out of it)
        delete c;
        return PDF_ECUDA;
    }
    c->cover_threads = 256;
    c->cover_grid = (uint32_t)prop.multiProcessorCount;

    auto fail = [&](pdf_status st2) {
        c->segs.release();
        c->seg_off.release();
        c->mem.release();
        delete c;
        return st2;
    };
    // One device block: both plans' arrays.
    {
        PlanUpload up;
        const ResidentImage none;
        const bool reduced = rnet.n_gates() != 0;
        const PlanOffsets fo = up.add_plan(net, full, reduced ? none : image);
        const PlanOffsets ro = reduced ? up.add_plan(rnet, red, image) : PlanOffsets{};
        const PlanOffsets lo = out_of == kOutLive ? up.add_plan(lnet, live, limage) : PlanOffsets{};
        const size_t vo = up.add(value.data(), value.size());
        const WideSync rest{};
        const size_t so = up.add(&rest, sizeof rest);
        if (c->mem.ensure(up.bytes) != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(PDF_ENOMEM);
        }
        if (!up.copy(c->mem.as<unsigned char>())) {
            (void)cudaGetLastError();
            return fail(PDF_ECUDA);
        }
        c->stage.sync = reinterpret_cast<WideSync *>(c->mem.as<unsigned char>() + so);
        c->full.bind(full, net, reduced ? none : image, c->mem.as<unsigned char>(), fo);
        if (reduced) c->red.bind(red, rnet, image, c->mem.as<unsigned char>(), ro);
        if (out_of == kOutLive) c->live.bind(live, lnet, limage, c->mem.as<unsigned char>(), lo);
        c->out_plan = out_of == kOutLive ? &c->live : out_of == kOutRed ? &c->red : out_of == kOutFull ? &c->full : nullptr;
        c->value = reinterpret_cast<const int8_t *>(c->mem.as<unsigned char>() + vo);
        c->full.wide = wide_full;
        c->red.wide = wide_red;
        c->full.mean_width = (uint32_t)mean_width;
        if (reduced) c->red.mean_width = (uint32_t)mean_level(rnet);
        for (Plan *p : {&c->full, &c->red, &c->live, &c->tile_full.plan, &c->tile_red.plan}) {
            p->res.sms = (uint32_t)prop.multiProcessorCount;
            p->res.regs = kResidentRegs;  // its launch bound's
            p->res.smem_block = res_smem;
            p->res.smem_sm = (size_t)prop.sharedMemPerMultiprocessor;
        }
        for (auto *t : {&c->tile_full, &c->tile_red})
            if (t->wanted) {
                const uint32_t bw = t->opts.bw;
                t->opts = po;
                t->opts.bw = bw;
                t->net = std::move(t == &c->tile_full ? net : rnet);
            }
    }
    inf.tile_words = c->bw;
    inf.threads = c->full.threads;
    inf.max_pairs = o.max_pairs ? o.max_pairs : 65536;
    if (o.seg_len > 1) {
        const pdf_status sst = build_segments(c, nl, o.seg_len);
        if (sst != PDF_OK) {
            (void)cudaGetLastError();
            return fail(sst);
        }
    }
    inf.seg_len = c->seg_len;
    inf.n_segments = c->n_first();
    inf.device_bytes = c->mem.bytes + c->segs.bytes + c->seg_off.bytes;
    *out = c;
    return PDF_OK;
}

extern "C" pdf_status pdf_circuit_segments(const pdf_circuit *c, uint32_t *gates) {
    if (!c || !gates) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    if (c->seg_len <= 1) {
        for (uint32_t g = 0; g < c->info.n_gates; g++) gates[g] = g;
        return PDF_OK;
    }
    PDF_CUDA(cudaMemcpy(gates, c->segs.p, (size_t)c->n_segs * c->seg_len * 4, cudaMemcpyDeviceToHost));
    return PDF_OK;
}

extern "C" void pdf_circuit_destroy(pdf_circuit *c) {
    if (!c) return;
    DeviceGuard dg(c->device);
    c->stage.release();
    c->mem.release();
    c->tile_full.mem.release();
    c->tile_red.mem.release();
    c->segs.release();
    c->seg_off.release();
    // after a cudaFree, which waits for what may still write there
    if (c->host_err && cudaFreeHost(c->host_err) != cudaSuccess) (void)cudaGetLastError();
    delete c;
}

extern "C" pdf_status pdf_circuit_query(const pdf_circuit *c, pdf_circuit_info *info) {
    if (!c || !info) return PDF_EINVAL;
    *info = c->info;
    return PDF_OK;
}

// ---------------------------------------------------------------------------

extern "C" pdf_status pdf_state_create(pdf_circuit *c, pdf_state **out) {
    if (!c || !out) return PDF_EINVAL;
    *out = nullptr;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    pdf_state *s = new (std::nothrow) pdf_state();
    if (!s) return PDF_ENOMEM;
    s->c = c;
    s->device = c->device;
    const size_t G = c->n_first();  // first-detect entries: nets, or segments
    const size_t acc_off = (8 * G + 255) & ~(size_t)255;
    const size_t sync_off = acc_off + ((sizeof(DevAcc) + 255) & ~(size_t)255);
    if (s->mem.ensure(sync_off + sizeof(WideSync)) != cudaSuccess ||
        cudaHostAlloc(reinterpret_cast<void **>(&s->host_acc), 2 * sizeof(DevAcc), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(reinterpret_cast<void **>(&s->mirror), s->host_acc + 1, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        pdf_state_destroy(s);
        return PDF_ENOMEM;
    }
    std::memset(s->host_acc, 0, 2 * sizeof(DevAcc));
    s->first_x.p = s->mem.p;
    s->first_y.p = s->mem.as<uint32_t>() + G;
    s->acc.p = s->mem.as<unsigned char>() + acc_off;
    s->ws.sync = reinterpret_cast<WideSync *>(s->mem.as<unsigned char>() + sync_off);
    // cleared on a stream of its own: a device-wide sync here would wait for
    // every other circuit's work in flight (a server creates states while it
    // grades)
    cudaStream_t cs = nullptr;
    const bool ok = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) == cudaSuccess &&
                    cudaMemsetAsync(s->ws.sync, 0, sizeof(WideSync), cs) == cudaSuccess &&
                    launch_state_reset(s->first_x.as<uint32_t>(), 2 * G, s->acc.as<DevAcc>(), s->mirror, cs) ==
                        cudaSuccess &&
                    cudaStreamSynchronize(cs) == cudaSuccess;
    if (cs) cudaStreamDestroy(cs);
    if (!ok) {
        note_cuda_error(cudaGetLastError(), "pdf_state_create: clearing the state", __LINE__);
        pdf_state_destroy(s);
        return PDF_ECUDA;
    }
    *out = s;
    return PDF_OK;
}

extern "C" void pdf_state_destroy(pdf_state *s) {
    if (!s) return;
    DeviceGuard dg(s->device);
    prof_release(s->prof);
    prof_release(s->pool);
    s->ws.release();
    s->mem.release();
    if (s->host_acc && cudaFreeHost(s->host_acc) != cudaSuccess) (void)cudaGetLastError();
    delete s;
}

extern "C" pdf_status pdf_state_reset(pdf_state *s) {
    if (!s) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    const size_t G = s->c->n_first();
    PDF_CUDA(cudaDeviceSynchronize());
    PDF_CUDA(launch_state_reset(s->first_x.as<uint32_t>(), 2 * G, s->acc.as<DevAcc>(), s->mirror, nullptr));
    PDF_CUDA(cudaDeviceSynchronize());
    return PDF_OK;
}

extern "C" pdf_status pdf_state_reset_async(pdf_state *s, void *stream) {
    if (!s) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const size_t G = s->c->n_first();
    PDF_CUDA(launch_state_reset(s->first_x.as<uint32_t>(), 2 * G, s->acc.as<DevAcc>(), s->mirror, cs));
    return PDF_OK;
}

extern "C" pdf_status pdf_state_profile(pdf_state *s, int enable) {
    if (!s) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    std::lock_guard<std::mutex> lk(s->mu);
    PDF_CUDA(cudaDeviceSynchronize());
    for (auto &p : s->prof) s->pool.push_back(p);
    s->prof.clear();
    s->profiling = enable != 0;
    return PDF_OK;
}

extern "C" pdf_status pdf_state_profile_read(pdf_state *s, double *ms, uint32_t *calls) {
    if (!s || !ms) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    std::lock_guard<std::mutex> lk(s->mu);
    ms[0] = ms[1] = ms[2] = 0;
    for (auto &p : s->prof) {
        PDF_CUDA(cudaEventSynchronize(p.ev[3]));
        float a = 0, b = 0, c = 0;
        PDF_CUDA(cudaEventElapsedTime(&a, p.ev[0], p.ev[1]));
        PDF_CUDA(cudaEventElapsedTime(&b, p.ev[2], p.ev[3]));
        PDF_CUDA(cudaEventElapsedTime(&c, p.ev[0], p.ev[3]));
        ms[0] += a;
        ms[1] += b;
        ms[2] += c;
    }
    if (calls) *calls = (uint32_t)s->prof.size();
    return PDF_OK;
}

extern "C" pdf_status pdf_state_snapshot(pdf_state *s, uint32_t *first_x, uint32_t *first_y,
                                         pdf_totals *tot) {
    if (!s) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    const size_t G = s->c->n_first();
    PDF_CUDA(cudaDeviceSynchronize());
    if (first_x) PDF_CUDA(cudaMemcpy(first_x, s->first_x.p, 4 * G, cudaMemcpyDeviceToHost));
    if (first_y) PDF_CUDA(cudaMemcpy(first_y, s->first_y.p, 4 * G, cudaMemcpyDeviceToHost));
    DevAcc h{};
    PDF_CUDA(cudaMemcpy(&h, s->acc.p, sizeof h, cudaMemcpyDeviceToHost));
    if (tot) {
        tot->lo = h.total_lo;
        tot->hi = h.total_hi;
        tot->pairs = h.pairs;
        tot->flags = h.flags;
        tot->reserved = 0;
    }
    return err_status(h.err);
}

extern "C" pdf_status pdf_state_snapshot_on(pdf_state *s, uint32_t *first_x, uint32_t *first_y, pdf_totals *tot,
                                            void *stream) {
    if (!s) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    const size_t G = s->c->n_first();
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    if (first_x) PDF_CUDA(cudaMemcpyAsync(first_x, s->first_x.p, 4 * G, cudaMemcpyDeviceToHost, cs));
    if (first_y) PDF_CUDA(cudaMemcpyAsync(first_y, s->first_y.p, 4 * G, cudaMemcpyDeviceToHost, cs));
    // the mirror holds the accumulators, unless a batch is marked and not yet
    // counted (its marking may have left an error there)
    const bool fetch = s->pending;
    if (fetch) PDF_CUDA(cudaMemcpyAsync(s->host_acc, s->acc.p, sizeof(DevAcc), cudaMemcpyDeviceToHost, cs));
    PDF_CUDA(cudaStreamSynchronize(cs));
    const DevAcc h = s->host_acc[fetch ? 0 : 1];
    if (tot) {
        tot->lo = h.total_lo;
        tot->hi = h.total_hi;
        tot->pairs = h.pairs;
        tot->flags = h.flags;
        tot->reserved = 0;
    }
    return err_status(h.err);
}

extern "C" pdf_status pdf_state_restore(pdf_state *s, const uint32_t *first_x,
                                        const uint32_t *first_y, const pdf_totals *tot) {
    if (!s || !first_x || !first_y || !tot) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    const size_t G = s->c->n_first();
    PDF_CUDA(cudaDeviceSynchronize());
    PDF_CUDA(cudaMemcpy(s->first_x.p, first_x, 4 * G, cudaMemcpyHostToDevice));
    PDF_CUDA(cudaMemcpy(s->first_y.p, first_y, 4 * G, cudaMemcpyHostToDevice));
    DevAcc h{};
    h.total_lo = tot->lo;
    h.total_hi = tot->hi;
    h.pairs = tot->pairs;
    h.flags = tot->flags;
    PDF_CUDA(cudaMemcpy(s->acc.p, &h, sizeof h, cudaMemcpyHostToDevice));
    PDF_CUDA(cudaDeviceSynchronize());
    s->host_acc[1] = h;
    return PDF_OK;
}

// ---------------------------------------------------------------------------

namespace {

pdf_status check_pairs(const pdf_circuit *c, const pdf_pairs *pr, uint64_t pair_base) {
    if (!pr || !pr->v || !pr->t) return PDF_EINVAL;
    if (pr->n_pairs == 0) return PDF_EINVAL;
    if (pr->ld < (pr->n_pairs + 31) / 32) return PDF_EINVAL;
    if (pair_base + pr->n_pairs > 0xFFFFFFFFull) return PDF_EINVAL;  // pair ids are uint32, ~0 = none
    (void)c;
    return PDF_OK;
}

// Slots of the spill cover for circuits of n gates: 2 x n u128 each, up to
// 16 MiB in all, at least one.
uint32_t spill_slots(uint64_t n, uint64_t *slot) {
    *slot = 2 * n * 16;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(16, (16ull << 20) / *slot));
}

// A walk's part of the workspace, W words of pairs: one block, since each
// allocation costs a new state's first call 20 to 300 us.  A resident walk's
// column block depends on W, so its share is sized for every smaller W too.
struct Scratch {
    uint32_t *nzb = nullptr, *maxlvl = nullptr;
    uint32_t *nzb_fine = nullptr, *maxlvl_fine = nullptr;  // the cover's bitmaps per kLaneCoverWords words
    uint32_t *active = nullptr, *active_list = nullptr;    // bitmap [W], then the count; <= 2 pairs per gate
    uint32_t *mid_list = nullptr;                          // pairs for the cover's large table
    uint32_t *over_list = nullptr;                         // pairs for the spill cover
    unsigned char *spill = nullptr;                        // and its per-net (h, c) slots
    uint8_t *flags = nullptr;                              // wide kernel: mark flags per (segment, gate)
    size_t bytes = 0;
};
Scratch scratch_of(const pdf_circuit *c, const Walk &k, uint64_t W, unsigned char *base) {
    const Plan &p = *k.p;
    const uint64_t n_blocks = k.resident ? W : (W + k.bw - 1) / k.bw;
    const uint64_t bm_bytes = (uint64_t)(p.n_gates + 31) / 32 * 4;
    Scratch x;
    if (k.out == RES_SIM) return x;
    const auto take = [&](auto *&q, uint64_t n) {
        q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(base + x.bytes);
        x.bytes += (n + 255) & ~(uint64_t)255;
    };
    if (k.wide) {
        // (segments of one chunk are the most there can be, for either width)
        take(x.flags, (uint64_t)p.n_gates * ((W + 31) / 32));
    } else {
        take(x.nzb, n_blocks * bm_bytes);
        take(x.maxlvl, n_blocks * 4);
    }
    if (k.fine()) {
        const uint64_t nf = n_blocks * (k.bw / kLaneCoverWords);
        take(x.nzb_fine, nf * bm_bytes);
        take(x.maxlvl_fine, nf * 4);
    }
    take(x.active, W * 4 + 16);
    const uint64_t list = std::min<uint64_t>(W * 32, 2 * std::max<uint64_t>(c->n_first(), c->info.n_gates)) * 4;
    take(x.active_list, list);
    take(x.mid_list, list);
    // A pair can mark more nets than the cover's table holds only when the
    // walk has more gates than that; its count then goes through the spill
    // cover.
    if (p.n_gates > c->hash_cap) {
        uint64_t slot;
        const uint32_t slots = spill_slots(p.n_gates, &slot);
        take(x.over_list, list);
        take(x.spill, slots * slot);
    }
    return x;
}

// A resident walk keeps V and T on chip: marks only in the workspace, of its own gates.
uint64_t resident_mark_words(const Walk &k, uint64_t W) {
    return k.out == RES_SIM ? 0 : (uint64_t)k.p->n_gates * ((W + 7) / 8 * 8);
}
uint64_t out_pitch(uint64_t W) { return (W + 3) / 4 * 4; }  // of planes that it writes into the workspace
// Words of the workspace's planes; `need`: the caller gives none that the walk can write.
uint64_t ws_plane_words(const pdf_circuit *c, const Walk &k, uint64_t W, bool need) {
    if (!k.resident) return need ? 3 * (uint64_t)k.p->n_gates * ((W + k.bw - 1) / k.bw * k.bw) : 0;
    return resident_mark_words(k, W) + (k.out != RES_LEAN && need ? 3 * (uint64_t)c->info.n_gates * out_pitch(W) : 0);
}

// What walks over W words of pairs take of a workspace.
struct WsNeed {
    uint64_t scratch = 0, planes = 0;  // bytes
    WsNeed &with(const pdf_circuit *c, const Walk &k, uint64_t W, bool need_planes) {
        scratch = std::max<uint64_t>(scratch, scratch_of(c, k, W, nullptr).bytes);
        planes = std::max(planes, ws_plane_words(c, k, W, need_planes) * 4);
        return *this;
    }
    // ... and what the resident walk takes that calls over fewer words may have
    // instead (calls within a workspace allocate nothing)
    WsNeed &lean(const pdf_circuit *c, const Walk &k, uint64_t W) {
        if (!k.resident && c->lean().image) {
            const Plan &p = c->lean();
            const uint64_t w = std::min<uint64_t>(W, resident_words(pdf_circuit::resident_walk(p, W, RES_LEAN).rs, p.res.sms));
            with(c, pdf_circuit::resident_walk(p, w, RES_LEAN), w, true);
        }
        return with(c, k, W, true);
    }
    WsNeed &out(const pdf_circuit *c, const Walk &k, uint64_t W, int out, bool need_planes) {
        if (!k.resident && c->out_plan) with(c, pdf_circuit::resident_walk(*c->out_plan, W, out), W, need_planes);
        return with(c, k, W, need_planes);
    }
    // every walk of a batch (sized without building the plan at the tile)
    WsNeed &batch(const pdf_circuit *c, uint64_t W) {
        const Plan &p = c->lean();
        if (p.image) with(c, pdf_circuit::resident_walk(p, W, RES_LEAN), W, true);
        Walk k;
        k.p = &p;
        for (uint32_t bw : {p.bw, c->tile_red.wanted ? c->tile_red.opts.bw : c->bw}) {
            k.bw = bw;
            with(c, k, W, true);
        }
        return *this;
    }
};

// Sizes the workspace.  A block that is too small and held stays allocated
// until nobody holds it.
pdf_status ensure_ws(pdf_circuit *c, const WsNeed &need, Workspace &ws, uint64_t W) {
    KeptBlocks *kept = &ws.kept;
    if (ws.scratch.bytes < need.scratch || ws.planes.bytes < need.planes) ws.sweep();  // (this call allocates anyway)
    if (c->seg_len > 1) {
        // (net, pair) entries: at most N per first pair of a segment, two per
        // segment, and one per (net, pair); a table at least twice that
        const uint64_t most = std::min<uint64_t>(2 * c->n_segs * c->seg_len, (uint64_t)c->info.n_gates * W * 32);
        uint64_t cap = 1024;
        while (cap < 2 * most && cap < (1ull << 27)) cap <<= 1;
        if (ws.seg_first.bytes < cap * 8) {  // (the block itself: a growth that failed has left none)
            PDF_CUDA(ws.seg_first.ensure(cap * 8, kept));
            ws.seg_first_mask = cap - 1;
        }
    }
    PDF_CUDA(ws.scratch.ensure(need.scratch, kept));
    PDF_CUDA(ws.planes.ensure(need.planes, kept));
    return PDF_OK;
}
pdf_status ensure_ws(pdf_circuit *c, const Walk &k, Workspace &ws, uint64_t W, bool need_planes) {
    return ensure_ws(c, WsNeed{}.with(c, k, W, need_planes), ws, W);
}
Scratch ws_scratch(const pdf_circuit *c, const Walk &k, const Workspace &ws, uint64_t W) {
    return scratch_of(c, k, W, ws.scratch.as<unsigned char>());
}
void use_scratch(FwdArgs &a, const Scratch &x) {
    a.nzb = x.nzb;
    a.blk_maxlvl = x.maxlvl;
    a.nzb_fine = x.nzb_fine;
    a.maxlvl_fine = x.maxlvl_fine;
}

// The workspace's planes for a walk over W words (after ensure_ws).
void use_ws_planes(FwdArgs &a, const Walk &k, const Workspace &ws, uint64_t W) {
    a.ld = (W + k.bw - 1) / k.bw * k.bw;
    if (k.resident) {
        a.M = ws.planes.as<uint32_t>();
        return;
    }
    a.V = ws.planes.as<uint32_t>();
    a.T = a.V + k.p->n_gates * a.ld;
    a.M = a.T + k.p->n_gates * a.ld;
}

// The planes that a resident walk writes: the caller's (direct), or the workspace's.
void use_out_planes(FwdArgs &a, const pdf_circuit *c, const Walk &k, const Workspace &ws, uint64_t W, bool direct,
                    uint32_t *v, uint32_t *t, uint32_t *m, uint64_t ld) {
    if (!direct) {
        ld = out_pitch(W);
        v = ws.planes.as<uint32_t>() + resident_mark_words(k, W);
        t = v + c->info.n_gates * ld;
        m = k.out == RES_SIM ? nullptr : t + c->info.n_gates * ld;
    }
    a.out_v = v;
    a.out_t = t;
    a.out_m = m;
    a.out_ld = ld;
}

FwdArgs base_fwd(pdf_circuit *c, const Walk &k, uint64_t n_pairs) {
    const Plan &p = *k.p;
    FwdArgs a{};
    a.c = p.dc;
    a.pieces = p.pieces;
    a.n_pieces = p.n_pieces;
    a.cap = p.cap;
    a.ecap = p.ecap;
    a.n_pairs = n_pairs;
    a.W = (uint32_t)((n_pairs + 31) / 32);
    a.store_all = 1;
    a.bm_words = (p.n_gates + 31) / 32;
    a.bm_shared = p.bm_shared;
    a.far_ids = p.far_ids;
    a.farcap = p.farcap;
    a.ring_gates = p.ring;
    a.ring2_gates = p.ring2;
    a.off_ring = p.off_ring;
    a.off_rec = p.off_rec;
    a.off_edge = p.off_edge;
    a.off_fid = p.off_fid;
    a.off_bm = p.off_bm;
    a.off_pbits = p.off_pbits;
    a.off_mbar = p.off_mbar;
    a.err = c->err;
    a.wait_polls = c->wait_polls;
    if (k.resident) {
        a.image = p.image;
        a.image_bytes = p.res.image_bytes;
        a.image_ids = p.image_ids;
        a.per = k.rs.per;
        a.n_blocks = k.rs.blocks;
        a.off_edge = p.off_edge_im;
        a.off_fid = p.off_lvl_im;
        a.off_ring = k.rs.off_vt;
        a.off_rec = k.rs.off_m;
        a.off_bm = k.rs.off_bm;
        a.off_mbar = k.rs.off_mbar;
    }
    return a;
}

cudaError_t launch_walk(const pdf_circuit *c, const Walk &k0, Workspace &ws, const FwdArgs &a, int mode,
                        cudaStream_t cs) {
    Walk k = k0;
    const Plan &p = *k.p;
    if (k.wide) {
        // two words per lane need rows and inputs that start on 8 bytes
        const auto even = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0; };
        const bool two = a.ld % 2 == 0 && even(a.V) && even(a.T) && even(a.M) &&
                         (mode == FWD_MARK || (a.pi_ld % 2 == 0 && even(a.pi_v) && even(a.pi_t)));
        if (!two) {
            k.cps = 0;
            c->wide_shape(k, a.W, 1);
        }
        WideArgs wa{};
        wa.flags = ws_scratch(c, k0, ws, a.W).flags;
        wa.sync = ws.sync;
        wa.cps = k.cps;
        wa.nseg = k.nseg;
        wa.chunks = k.chunks;
        return launch_wide(a, wa, mode, c->mark_mode, k.wide, p.res.sms, cs);
    }
    if (k.resident && k.out != RES_LEAN) {
        const cudaError_t e = launch_fill_planes(c->value, c->info.n_gates, a.n_pairs, a.out_v, a.out_t, a.out_m,
                                                 a.out_ld, p.res.sms, cs);
        if (e != cudaSuccess) return e;
    }
    if (k.resident) return launch_resident(a, c->mark_mode, k.out, k.bw, k.rs.ctas, k.rs.threads, k.rs.smem, cs);
    if (lane_tile(k.bw)) return launch_lanes(a, mode, c->mark_mode, k.bw, p.threads, p.fwd_smem, cs);
    return launch_forward(a, mode, c->mark_mode, k.bw, p.threads, p.fwd_smem, cs);
}

// The error word of the circuit's stage calls (pdf_sim, pdf_mark): read after
// the call's work is done, then cleared, so that an expired wait is reported by
// the call that met it and by no later one.
pdf_status open_circuit_err(pdf_circuit *c) {
    if (c->host_err) return PDF_OK;
    PDF_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&c->host_err), 64, cudaHostAllocMapped));
    *c->host_err = 0;
    const cudaError_t e = cudaHostGetDevicePointer(reinterpret_cast<void **>(&c->err), c->host_err, 0);
    if (e != cudaSuccess) {
        cudaFreeHost(c->host_err);
        c->host_err = nullptr;
    }
    PDF_CUDA(e);
    return PDF_OK;
}
pdf_status take_circuit_err(pdf_circuit *c, cudaStream_t cs) {
    PDF_CUDA(cudaStreamSynchronize(cs));
    const unsigned int e = *reinterpret_cast<volatile uint32_t *>(c->host_err);
    *c->host_err = 0;
    return err_status(e);
}

// How many first-detecting pairs skip the cover's small table: up to one per SM,
// which the large table takes side by side too, where pairs often do not fit the
// small one and would be walked twice (netlists of 2^16 gates or more); up to two
// where they mostly do not (2^18 gates, the FIXED non-robust table).  Measured
// (cover kernels, us; through both tables and at once): 200,000 gates, 100 pairs
// 90 and 79; 1,000,000 gates, 32 pairs 459 and 211, 256 pairs 591 and 485; FIXED
// non-robust, 20,000 gates, 32 pairs 211 and 139, 247 pairs 364 and 330, 477 pairs
// 565 and 585 (one table).  Where they fit, the second pass is a launch too many:
// 20,000 gates with segments, a whole call 196 and 200; FIXED robust, 60,000
// gates, 238 pairs 103 and 160.
uint32_t cover_few(const pdf_circuit *c, const Plan &p) {
    if (c->mark_mode == PDF_MARK_FIXED_NONROBUST || p.n_gates >= 1u << 18) return 2 * c->cover_grid;
    return p.n_gates >= 1u << 16 ? c->cover_grid : 0;
}

CoverArgs base_cover(pdf_circuit *c, const Walk &k, Workspace &ws, const uint32_t *M, uint64_t ld, uint64_t n_pairs,
                     uint32_t pair_base, const uint32_t *fx, const uint32_t *fy, DevAcc *acc) {
    const Plan &p = *k.p;
    CoverArgs a{};
    a.c = p.dc;
    a.M = M;
    a.ld = ld;
    // a lane walk's cover reads bitmaps per 8 words of its column blocks
    // (fewer candidate nets per pair than the whole block's)
    const bool fine = k.fine();
    const Scratch x = ws_scratch(c, k, ws, (n_pairs + 31) / 32);
    a.nzb = fine ? x.nzb_fine : x.nzb;
    a.blk_maxlvl = fine ? x.maxlvl_fine : x.maxlvl;
    a.bm_words = (p.n_gates + 31) / 32;
    a.bw = fine ? kLaneCoverWords : k.bw;
    a.first_x = fx;
    a.first_y = fy;
    a.n_pairs = n_pairs;
    a.pair_base = pair_base;
    a.active = x.active;
    a.active_count = a.active + (n_pairs + 31) / 32;
    a.active_list = x.active_list;
    a.acc = acc;
    a.hash_cap = c->hash_cap;
    a.mid_list = x.mid_list;
    a.small_cap = c->small_cap;
    a.few = cover_few(c, p);
    a.over_list = x.over_list;
    a.spill = x.spill;
    uint64_t slot;
    a.spill_slots = p.n_gates > c->hash_cap ? spill_slots(p.n_gates, &slot) : 0;
    a.seg = c->seg_args();
    if (c->seg_len > 1) {
        a.seg_first = ws.seg_first.as<unsigned long long>();
        a.seg_first_mask = ws.seg_first_mask;
    }
    return a;
}

// Device pointers of the pairs (staging host pairs through the workspace).
// True when (ptr, ld) can be used by the kernels directly: rows of ld words,
// ld a multiple of the tile width and below 2^30 (row pitches in bytes fit
// 32 bits), every row long enough for whole tiles, and 16-byte aligned base
// addresses.
bool planes_fit(const pdf_circuit *c, uint64_t W, uint64_t ld, std::initializer_list<const void *> ptrs) {
    const uint64_t Wp = (W + c->bw - 1) / c->bw * c->bw;
    if (ld < Wp || ld % c->bw || ld >= (1ull << 30)) return false;
    for (const void *p : ptrs)
        if (!p || (reinterpret_cast<uintptr_t>(p) & 15)) return false;
    return true;
}

// The same for output and stage planes on walk k: the wide and the resident
// kernel take any pitch and word-aligned rows.
bool planes_fit(const pdf_circuit *c, const Walk &k, uint64_t W, uint64_t ld, std::initializer_list<const void *> ptrs) {
    if (!k.wide && !k.resident) return planes_fit(c, W, ld, ptrs);
    if (ld < W || ld >= (1ull << 30)) return false;
    for (const void *p : ptrs)
        if (!p || (reinterpret_cast<uintptr_t>(p) & 3)) return false;
    return true;
}

// Device pointers of the pairs, staging them through the workspace when
// they are host memory or not in the kernels' layout.
// A resident walk reads them word by word, at any pitch.
pdf_status stage_pairs(pdf_circuit *c, const Walk &k, Workspace &ws, const pdf_pairs *pr, const uint32_t **v,
                       const uint32_t **t, uint64_t *ld, cudaStream_t st) {
    const uint64_t W = (pr->n_pairs + 31) / 32, npi = c->info.n_pi;
    const bool words = ((reinterpret_cast<uintptr_t>(pr->v) | reinterpret_cast<uintptr_t>(pr->t)) & 3) == 0;
    if (pr->on_device && pr->ld < (1ull << 30) && (k.resident || k.wide ? words : planes_fit(c, W, pr->ld, {pr->v, pr->t}))) {
        *v = pr->v;
        *t = pr->t;
        *ld = pr->ld;
        return PDF_OK;
    }
    const uint64_t Wp = k.resident ? W : (W + c->bw - 1) / c->bw * c->bw;
    PDF_CUDA(ws.pi.ensure(2 * npi * ((W + c->bw - 1) / c->bw * c->bw) * 4, &ws.kept));
    uint32_t *dv = ws.pi.as<uint32_t>(), *dt = dv + npi * Wp;
    const cudaMemcpyKind kind = pr->on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    if (pr->ld == Wp) {  // rows already at the device pitch: one contiguous copy per plane
        PDF_CUDA(cudaMemcpyAsync(dv, pr->v, npi * Wp * 4, kind, st));
        PDF_CUDA(cudaMemcpyAsync(dt, pr->t, npi * Wp * 4, kind, st));
    } else {
        PDF_CUDA(cudaMemcpy2DAsync(dv, Wp * 4, pr->v, pr->ld * 4, W * 4, npi, kind, st));
        PDF_CUDA(cudaMemcpy2DAsync(dt, Wp * 4, pr->t, pr->ld * 4, W * 4, npi, kind, st));
    }
    *v = dv;
    *t = dt;
    *ld = Wp;
    return PDF_OK;
}

pdf_status copy_plane_out(uint32_t *dst, uint64_t dst_ld, int dst_dev, const uint32_t *src,
                          uint64_t src_ld, uint64_t W, uint64_t G, cudaStream_t st) {
    if (!dst) return PDF_OK;
    if (dst_ld < W) return PDF_EINVAL;
    PDF_CUDA(cudaMemcpy2DAsync(dst, dst_ld * 4, src, src_ld * 4, W * 4, G,
                               dst_dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st));
    return PDF_OK;
}

}  // namespace

namespace {

// First half of a grading call: sim, mark, prune and merge into the state.
// Records what the second half needs in the state.
pdf_status grade_mark_locked(pdf_circuit *c, pdf_state *s, const pdf_pairs *pr, uint64_t pair_base,
                             const pdf_outputs *out, cudaStream_t cs) {
    const uint64_t n = pr->n_pairs, W = (n + 31) / 32, G = c->info.n_gates;
    // with no plane asked for, only what the marks depend on is evaluated,
    // and only the rows read back are written
    const bool planes = out && (out->sim_v || out->sim_t || out->mark);
    const Walk k = planes ? c->planes_walk(W) : c->lean_walk(W);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    PDF_CUDA(cudaStreamIsCapturing(cs, &cap));
    const Plan &p = *k.p;
    const bool direct = out && out->on_device && planes_fit(c, k, W, out->ld, {out->sim_v, out->sim_t, out->mark});
    WsNeed need;
    if (planes) need.out(c, k, W, RES_PLANES, !direct);
    else need.lean(c, k, W);
    pdf_status st = ensure_ws(c, need, s->ws, W);
    if (st != PDF_OK) return st;
    const uint32_t *pv, *pt;
    uint64_t pld;
    st = stage_pairs(c, k, s->ws, pr, &pv, &pt, &pld, cs);
    if (st != PDF_OK) return st;
    if (cap != cudaStreamCaptureStatusNone) s->ws.hold_for_graph();  // it will have its addresses

    FwdArgs a = base_fwd(c, k, n);
    a.pi_v = pv;
    a.pi_t = pt;
    a.pi_ld = pld;
    a.store_all = planes ? 1u : 0u;
    a.in_pieces = planes ? 0u : p.in_pieces;
    if (k.resident || !direct) use_ws_planes(a, k, s->ws, W);
    if (k.out == RES_PLANES) {
        use_out_planes(a, c, k, s->ws, W, direct, out->sim_v, out->sim_t, out->mark, out->ld);
    } else if (direct) {
        a.V = out->sim_v;
        a.T = out->sim_t;
        a.M = out->mark;
        a.ld = out->ld;
    }
    const Scratch x = ws_scratch(c, k, s->ws, W);
    use_scratch(a, x);
    // with segments the state holds per-segment ids, merged after the kernel
    a.first_x = c->seg_len > 1 ? nullptr : s->first_x.as<uint32_t>();
    a.first_y = c->seg_len > 1 ? nullptr : s->first_y.as<uint32_t>();
    a.pair_base = (uint32_t)pair_base;
    DevAcc *acc = s->acc.as<DevAcc>();
    a.err = &acc->err;
    s->pe = nullptr;
    if (s->profiling) {
        ProfEvents pe{};
        if (!s->pool.empty()) {
            pe = s->pool.back();
            s->pool.pop_back();
        } else {
            for (auto &e : pe.ev) PDF_CUDA(cudaEventCreate(&e));
        }
        s->prof.push_back(pe);
        s->pe = &s->prof.back();
        PDF_CUDA(cudaEventRecord(s->pe->ev[0], cs));
    }
    // the forward kernel also clears the batch count and the cover's active pairs
    a.acc = acc;
    a.active = x.active;
    PDF_CUDA(launch_walk(c, k, s->ws, a, FWD_FUSED, cs));
    if (c->seg_len > 1) {
        SegMergeArgs sm{};
        sm.seg = c->seg_args();
        sm.V = a.V;
        sm.M = a.M;
        sm.ld = a.ld;
        sm.nzb = k.fine() ? a.nzb_fine : a.nzb;
        sm.bm_words = a.bm_words;
        sm.bw = k.fine() ? kLaneCoverWords : p.bw;
        sm.W = (uint32_t)W;
        sm.pair_base = (uint32_t)pair_base;
        sm.first_x = s->first_x.as<uint32_t>();
        sm.first_y = s->first_y.as<uint32_t>();
        PDF_CUDA(launch_seg_merge(sm, (uint32_t)((W + sm.bw - 1) / sm.bw), cs));
    }
    if (s->pe) PDF_CUDA(cudaEventRecord(s->pe->ev[1], cs));
    if (out && !direct) {
        const bool o = k.out == RES_PLANES;
        const uint64_t ld = o ? a.out_ld : a.ld;
        st = copy_plane_out(out->sim_v, out->ld, out->on_device, o ? a.out_v : a.V, ld, W, G, cs);
        if (st == PDF_OK) st = copy_plane_out(out->sim_t, out->ld, out->on_device, o ? a.out_t : a.T, ld, W, G, cs);
        if (st == PDF_OK) st = copy_plane_out(out->mark, out->ld, out->on_device, o ? a.out_m : a.M, ld, W, G, cs);
        if (st != PDF_OK) return st;
    }
    s->pend_walk = k;
    s->pend_M = a.M;
    s->pend_ld = a.ld;
    s->pend_n = n;
    s->pend_base = pair_base;
    s->pending = true;
    return PDF_OK;
}

// Second half: count the covered paths of the marked batch against the
// state's first-detect ids and add them to the total.
pdf_status grade_cover_locked(pdf_circuit *c, pdf_state *s, cudaStream_t cs) {
    if (!s->pending) return PDF_EINVAL;
    s->pending = false;
    DevAcc *acc = s->acc.as<DevAcc>();
    const uint32_t base = (uint32_t)s->pend_base;
    CoverArgs ca = base_cover(c, s->pend_walk, s->ws, s->pend_M, s->pend_ld, s->pend_n, base, s->first_x.as<uint32_t>(),
                              s->first_y.as<uint32_t>(), acc);
    ca.mirror = s->mirror;
    if (s->pe) PDF_CUDA(cudaEventRecord(s->pe->ev[2], cs));  // cover starts (after any exchange)
    PDF_CUDA(launch_cover(ca, c->cover_grid, c->cover_threads, false, cs));  // closes the batch
    if (s->pe) {
        PDF_CUDA(cudaEventRecord(s->pe->ev[3], cs));
        s->pe = nullptr;
    }
    return PDF_OK;
}

}  // namespace

extern "C" pdf_status pdf_grade_mark_async(pdf_circuit *c, pdf_state *s, const pdf_pairs *pr,
                                           uint64_t pair_base, const pdf_outputs *out, void *stream) {
    if (!c || !s || s->c != c) return PDF_EINVAL;
    pdf_status st = check_pairs(c, pr, pair_base);
    if (st != PDF_OK) return st;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    std::lock_guard<std::mutex> lk(s->mu);
    return grade_mark_locked(c, s, pr, pair_base, out, static_cast<cudaStream_t>(stream));
}

extern "C" pdf_status pdf_grade_cover_async(pdf_circuit *c, pdf_state *s, void *stream) {
    if (!c || !s || s->c != c) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    std::lock_guard<std::mutex> lk(s->mu);
    return grade_cover_locked(c, s, static_cast<cudaStream_t>(stream));
}

extern "C" pdf_status pdf_grade_async(pdf_circuit *c, pdf_state *s, const pdf_pairs *pr,
                                      uint64_t pair_base, const pdf_outputs *out, void *stream) {
    if (!c || !s || s->c != c) return PDF_EINVAL;
    pdf_status st = check_pairs(c, pr, pair_base);
    if (st != PDF_OK) return st;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lk(s->mu);
    st = grade_mark_locked(c, s, pr, pair_base, out, cs);
    if (st != PDF_OK) return st;
    return grade_cover_locked(c, s, cs);
}

// Whether [x, end) lies in one device allocation (0.2 us; a second copy takes 3).
static bool one_allocation(uintptr_t x, uintptr_t end) {
    using Range = CUresult (*)(CUdeviceptr *, size_t *, CUdeviceptr);
    static const Range range = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Range>(f);
    }();
    CUdeviceptr base = 0;
    size_t size = 0;
    return range && range(&base, &size, x) == CUDA_SUCCESS && end <= base + size;
}

extern "C" pdf_status pdf_state_first_copy(pdf_state *s, uint32_t *first_x, uint32_t *first_y, int to_state,
                                           void *stream) {
    if (!s || !first_x || !first_y) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const size_t bytes = 4 * (size_t)s->c->n_first();
    uint32_t *sx = s->first_x.as<uint32_t>(), *sy = s->first_y.as<uint32_t>();
    // the state's two arrays are rows of one block, and so are the caller's
    // when the second lies past the first in one allocation: one copy of two rows
    const uintptr_t x = reinterpret_cast<uintptr_t>(first_x), y = reinterpret_cast<uintptr_t>(first_y);
    if (y >= x + bytes && y - x < (1ull << 31) && one_allocation(x, y + bytes)) {
        if (to_state) PDF_CUDA(cudaMemcpy2DAsync(sx, bytes, first_x, y - x, bytes, 2, cudaMemcpyDeviceToDevice, cs));
        else PDF_CUDA(cudaMemcpy2DAsync(first_x, y - x, sx, bytes, bytes, 2, cudaMemcpyDeviceToDevice, cs));
    } else if (to_state) {
        PDF_CUDA(cudaMemcpyAsync(sx, first_x, bytes, cudaMemcpyDeviceToDevice, cs));
        PDF_CUDA(cudaMemcpyAsync(sy, first_y, bytes, cudaMemcpyDeviceToDevice, cs));
    } else {
        PDF_CUDA(cudaMemcpyAsync(first_x, sx, bytes, cudaMemcpyDeviceToDevice, cs));
        PDF_CUDA(cudaMemcpyAsync(first_y, sy, bytes, cudaMemcpyDeviceToDevice, cs));
    }
    return PDF_OK;
}

extern "C" pdf_status pdf_grade(pdf_circuit *c, pdf_state *s, const pdf_pairs *pr, uint64_t pair_base,
                                const pdf_outputs *out, pdf_totals *batch, void *stream) {
    pdf_status st = pdf_grade_async(c, s, pr, pair_base, out, stream);
    if (st != PDF_OK) return st;
    DeviceGuard dg(c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    PDF_CUDA(cudaStreamSynchronize(cs));
    const DevAcc h = s->host_acc[1];  // left there by the cover
    if (batch) {
        batch->lo = h.batch_lo;
        batch->hi = h.batch_hi;
        batch->pairs = pr->n_pairs;
        batch->flags = h.batch_flags;
        batch->reserved = 0;
    }
    return err_status(h.err);
}

// ---- stage calls ----------------------------------------------------------

extern "C" pdf_status pdf_sim(pdf_circuit *c, const pdf_pairs *pr, uint32_t *sim_v, uint32_t *sim_t,
                              uint64_t ld, void *stream) {
    if (!c || !sim_v || !sim_t) return PDF_EINVAL;
    pdf_status st = check_pairs(c, pr, 0);
    if (st != PDF_OK) return st;
    const uint64_t W = (pr->n_pairs + 31) / 32, G = c->info.n_gates;
    if (ld < W) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lk(c->mu);
    if ((st = open_circuit_err(c)) != PDF_OK) return st;
    const Walk k = c->planes_walk(W, RES_SIM);
    const bool direct = planes_fit(c, k, W, ld, {sim_v, sim_t});
    st = ensure_ws(c, WsNeed{}.out(c, k, W, RES_SIM, !direct), c->stage, W);
    if (st != PDF_OK) return st;
    const uint32_t *pv, *pt;
    uint64_t pld;
    st = stage_pairs(c, k, c->stage, pr, &pv, &pt, &pld, cs);
    if (st != PDF_OK) return st;
    FwdArgs a = base_fwd(c, k, pr->n_pairs);
    a.pi_v = pv;
    a.pi_t = pt;
    a.pi_ld = pld;
    if (k.resident) {
        use_out_planes(a, c, k, c->stage, W, direct, sim_v, sim_t, nullptr, ld);
    } else if (direct) {
        a.V = sim_v;
        a.T = sim_t;
        a.ld = ld;
    } else {
        use_ws_planes(a, k, c->stage, W);
    }
    PDF_CUDA(launch_walk(c, k, c->stage, a, FWD_SIM, cs));
    if (!direct) {
        const uint32_t *v = k.resident ? a.out_v : a.V, *t = k.resident ? a.out_t : a.T;
        const uint64_t from = (k.resident ? a.out_ld : a.ld) * 4;
        PDF_CUDA(cudaMemcpy2DAsync(sim_v, ld * 4, v, from, W * 4, G, cudaMemcpyDeviceToDevice, cs));
        PDF_CUDA(cudaMemcpy2DAsync(sim_t, ld * 4, t, from, W * 4, G, cudaMemcpyDeviceToDevice, cs));
    }
    return take_circuit_err(c, cs);  // waits: the stage scratch is reused by the next stage call
}

namespace {

pdf_status mark_planes(pdf_circuit *c, const uint32_t *sim_v, const uint32_t *sim_t, uint32_t *mark,
                       uint64_t n_pairs, uint64_t ld, void *stream, bool prune) {
    if (!c || !sim_v || !sim_t || !mark || n_pairs == 0 || ld < (n_pairs + 31) / 32) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lk(c->mu);
    const uint64_t W = (n_pairs + 31) / 32, G = c->info.n_gates;
    const Walk k = c->full_walk(W);
    const bool direct = planes_fit(c, k, W, ld, {sim_v, sim_t, mark});
    pdf_status st = open_circuit_err(c);
    if (st == PDF_OK) st = ensure_ws(c, k, c->stage, W, !direct);
    if (st != PDF_OK) return st;
    FwdArgs a = base_fwd(c, k, n_pairs);
    if (direct) {
        a.V = const_cast<uint32_t *>(sim_v);
        a.T = const_cast<uint32_t *>(sim_t);
        a.M = mark;
        a.ld = ld;
    } else {
        use_ws_planes(a, k, c->stage, W);
        PDF_CUDA(cudaMemcpy2DAsync(a.V, a.ld * 4, sim_v, ld * 4, W * 4, G, cudaMemcpyDeviceToDevice, cs));
        PDF_CUDA(cudaMemcpy2DAsync(a.T, a.ld * 4, sim_t, ld * 4, W * 4, G, cudaMemcpyDeviceToDevice, cs));
    }
    use_scratch(a, ws_scratch(c, k, c->stage, W));
    a.no_prune = prune ? 0u : 1u;
    a.in_pieces = k.p->in_pieces;
    PDF_CUDA(launch_walk(c, k, c->stage, a, FWD_MARK, cs));
    if (!direct)
        PDF_CUDA(cudaMemcpy2DAsync(mark, ld * 4, a.M, a.ld * 4, W * 4, G, cudaMemcpyDeviceToDevice, cs));
    return take_circuit_err(c, cs);
}

}  // namespace

extern "C" pdf_status pdf_mark(pdf_circuit *c, const uint32_t *sim_v, const uint32_t *sim_t,
                               uint32_t *mark, uint64_t n_pairs, uint64_t ld, void *stream) {
    return mark_planes(c, sim_v, sim_t, mark, n_pairs, ld, stream, true);
}

extern "C" pdf_status pdf_mark_forward(pdf_circuit *c, const uint32_t *sim_v, const uint32_t *sim_t,
                                       uint32_t *mark, uint64_t n_pairs, uint64_t ld, void *stream) {
    return mark_planes(c, sim_v, sim_t, mark, n_pairs, ld, stream, false);
}

extern "C" pdf_status pdf_merge(pdf_circuit *c, pdf_state *s, const uint32_t *sim_v, const uint32_t *mark,
                                uint64_t n_pairs, uint64_t ld, uint64_t pair_base, void *stream) {
    if (!c || !s || s->c != c || !sim_v || !mark || n_pairs == 0 || ld < (n_pairs + 31) / 32)
        return PDF_EINVAL;
    if (pair_base + n_pairs > 0xFFFFFFFFull) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    if (c->seg_len > 1)
        PDF_CUDA(launch_seg_merge_dense(c->seg_args(), sim_v, mark, ld, n_pairs, (uint32_t)pair_base,
                                        s->first_x.as<uint32_t>(), s->first_y.as<uint32_t>(), cs));
    else
        PDF_CUDA(launch_merge_dense(c->full.dc, sim_v, mark, ld, n_pairs, (uint32_t)pair_base,
                                    s->first_x.as<uint32_t>(), s->first_y.as<uint32_t>(), cs));
    return PDF_OK;
}

namespace {

// pdf_cover, and with `counts` (host) the paths each primary input credits to
// each pair of the chunk.
pdf_status cover_chunk(pdf_circuit *c, pdf_state *s, const uint32_t *mark, uint64_t n_pairs, uint64_t ld,
                       uint64_t pair_base, uint64_t *counts, pdf_totals *chunk, cudaStream_t cs) {
    std::lock_guard<std::mutex> lk(s->mu);
    const uint64_t W = (n_pairs + 31) / 32;
    const Walk k = c->full_walk(W);
    pdf_status st = ensure_ws(c, k, s->ws, W, false);
    if (st != PDF_OK) return st;
    const size_t count_bytes = (size_t)c->info.n_pi * n_pairs * 16;
    if (counts) {
        PDF_CUDA(s->ws.pi_counts.ensure(count_bytes));
        PDF_CUDA(cudaMemsetAsync(s->ws.pi_counts.p, 0, count_bytes, cs));
    }
    DevAcc *acc = s->acc.as<DevAcc>();
    PDF_CUDA(launch_batch_begin(acc, cs));
    CoverArgs ca = base_cover(c, k, s->ws, mark, ld, n_pairs, (uint32_t)pair_base, s->first_x.as<uint32_t>(),
                              s->first_y.as<uint32_t>(), acc);
    // the bitmaps the cover reads, at its granularity, from the given marks
    PDF_CUDA(launch_bitmap_from_marks(c->full.dc, mark, ld, n_pairs, ca.bw, const_cast<uint32_t *>(ca.nzb),
                                      const_cast<uint32_t *>(ca.blk_maxlvl), ca.bm_words, cs));
    ca.mirror = s->mirror;
    if (counts) ca.pi_counts = s->ws.pi_counts.as<unsigned long long>();
    PDF_CUDA(launch_cover(ca, c->cover_grid, c->cover_threads, true, cs));  // closes the batch
    if (counts) PDF_CUDA(cudaMemcpyAsync(counts, s->ws.pi_counts.p, count_bytes, cudaMemcpyDeviceToHost, cs));
    PDF_CUDA(cudaStreamSynchronize(cs));
    const DevAcc h = s->host_acc[1];  // left there by the cover
    if (chunk) {
        chunk->lo = h.batch_lo;
        chunk->hi = h.batch_hi;
        chunk->pairs = n_pairs;
        chunk->flags = h.batch_flags;
        chunk->reserved = 0;
    }
    return err_status(h.err);
}

}  // namespace

extern "C" pdf_status pdf_cover(pdf_circuit *c, pdf_state *s, const uint32_t *mark, uint64_t n_pairs,
                                uint64_t ld, uint64_t pair_base, pdf_totals *chunk, void *stream) {
    if (!c || !s || s->c != c || !mark || n_pairs == 0 || ld < (n_pairs + 31) / 32) return PDF_EINVAL;
    if (pair_base + n_pairs > 0xFFFFFFFFull) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    return cover_chunk(c, s, mark, n_pairs, ld, pair_base, nullptr, chunk, static_cast<cudaStream_t>(stream));
}

extern "C" pdf_status pdf_cover_counts(pdf_circuit *c, pdf_state *s, const uint32_t *mark, uint64_t n_pairs,
                                       uint64_t ld, uint64_t pair_base, uint64_t *counts, pdf_totals *chunk,
                                       void *stream) {
    if (!c || !s || s->c != c || !mark || !counts || n_pairs == 0 || ld < (n_pairs + 31) / 32) return PDF_EINVAL;
    if (pair_base + n_pairs > 0xFFFFFFFFull) return PDF_EINVAL;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    return cover_chunk(c, s, mark, n_pairs, ld, pair_base, counts, chunk, static_cast<cudaStream_t>(stream));
}

// Allocation-free variant of pdf_cover: the same kernels, with their scratch
// carved from the fixed array g_cover_scratch (pdf_kernels.cu) instead of a
// workspace.  Allocates nothing, frees nothing.  The first call on a device
// looks the array's address up (noalloc_scratch).
extern "C" pdf_status pdf_cover_noalloc(pdf_circuit *c, const uint32_t *mark, uint64_t n_pairs, uint64_t ld,
                                        uint64_t pair_base, const uint32_t *first_x, const uint32_t *first_y,
                                        pdf_totals *chunk_total, void *stream) {
    if (!c || !mark || !first_x || !first_y || !chunk_total || n_pairs == 0 || ld < (n_pairs + 31) / 32)
        return PDF_EINVAL;
    if (c->seg_len > 1) return PDF_ENOTSUP;  // its fixed scratch holds no (net, pair) set
    if (pair_base + n_pairs > 0xFFFFFFFFull) return PDF_EINVAL;
    const uint64_t W = (n_pairs + 31) / 32, n_blocks = (W + c->bw - 1) / c->bw;
    const uint64_t bm_words = (c->info.n_gates + 31) / 32;
    auto a256 = [](uint64_t x) { return (x + 255) & ~(uint64_t)255; };
    const uint64_t o_maxlvl = a256(n_blocks * bm_words * 4);
    const uint64_t o_active = o_maxlvl + a256(n_blocks * 4);
    const uint64_t o_list = o_active + a256(W * 4 + 16);
    const uint64_t o_acc = o_list + a256(std::min<uint64_t>(W * 32, 2 * (uint64_t)c->info.n_gates) * 4);
    const uint64_t need = o_acc + a256(sizeof(DevAcc));
    if (need > kNoAllocScratchBytes) return PDF_ELIMIT;
    DeviceGuard dg(c->device);
    if (!dg.ok) return PDF_ECUDA;
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    unsigned char *base = nullptr;
    PDF_CUDA(noalloc_scratch(c->device, &base));
    uint32_t *nzb = reinterpret_cast<uint32_t *>(base);
    uint32_t *maxlvl = reinterpret_cast<uint32_t *>(base + o_maxlvl);
    uint32_t *active = reinterpret_cast<uint32_t *>(base + o_active);
    uint32_t *active_list = reinterpret_cast<uint32_t *>(base + o_list);
    DevAcc *acc = reinterpret_cast<DevAcc *>(base + o_acc);
    // the array keeps the previous call's contents: clear the accumulator
    PDF_CUDA(cudaMemsetAsync(acc, 0, sizeof(DevAcc), cs));
    PDF_CUDA(launch_batch_begin(acc, cs));
    PDF_CUDA(launch_bitmap_from_marks(c->full.dc, mark, ld, n_pairs, c->bw, nzb, maxlvl, (uint32_t)bm_words, cs));
    CoverArgs ca{};
    ca.c = c->full.dc;
    ca.M = mark;
    ca.ld = ld;
    ca.nzb = nzb;
    ca.blk_maxlvl = maxlvl;
    ca.bm_words = (uint32_t)bm_words;
    ca.bw = c->bw;
    ca.first_x = first_x;
    ca.first_y = first_y;
    ca.n_pairs = n_pairs;
    ca.pair_base = (uint32_t)pair_base;
    ca.active = active;
    ca.active_count = active + W;
    ca.active_list = active_list;
    ca.acc = acc;
    ca.hash_cap = c->hash_cap;
    PDF_CUDA(launch_cover(ca, c->cover_grid, c->cover_threads, true, cs));  // closes the batch
    DevAcc h{};
    PDF_CUDA(cudaMemcpyAsync(&h, acc, sizeof h, cudaMemcpyDeviceToHost, cs));
    PDF_CUDA(cudaStreamSynchronize(cs));
    chunk_total->lo = h.batch_lo;
    chunk_total->hi = h.batch_hi;
    chunk_total->pairs = n_pairs;
    chunk_total->flags = h.batch_flags;
    chunk_total->reserved = 0;
    return err_status(h.err);
}

// ---------------------------------------------------------------------------
// Batched grading.
// ---------------------------------------------------------------------------

struct pdf_batch {
    int device = 0;
    uint32_t small_cap = 0, small_per_sm = 0;  // the small-table cover: nets per pair, CTAs per SM
    std::vector<pdf_circuit *> circuits;
    std::vector<pdf_state *> states;
    BatchLaunch L{};
    DevBuf ctl;  // control word, arguments, prefixes and items in one block
    std::shared_ptr<const void> bound;  // token of this binding, in the blocks of its states' workspaces
    uint64_t gate_evals = 0, bytes = 0;
    cudaStream_t cap_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bool use_graph = true;
    bool ran = false;  // since it was built: the first run launches directly, the second captures
    // side streams and fork/join events of the forward launches per class
    cudaStream_t side[kMaxBatchClasses - 1] = {};
    cudaEvent_t fork = nullptr, join[kMaxBatchClasses - 1] = {};
    cudaStream_t up = nullptr;  // uploads of the control block
    cudaEvent_t uploaded = nullptr;
    bool wait_upload = false;   // the next run's stream still has to wait for it
    unsigned char *host_ctl = nullptr;  // mapped pinned staging of the control block
    size_t host_bytes = 0;
    cudaEvent_t prof[3] = {};  // pdf_batch_profile: pass start, forward joined, pass end
    bool profiling = false;
    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    void release() {
        for (auto &x : prof)
            if (x) cudaEventDestroy(x);
        for (auto &x : prof) x = nullptr;
        // the upload may not have been run, or a run that leaves its error word
        // there not have ended: the staging goes after the wait for the one and
        // the device block, whose cudaFree waits for the other
        if (uploaded && cudaEventSynchronize(uploaded) != cudaSuccess) (void)cudaGetLastError();
        ctl.release();
        if (host_ctl) cudaFreeHost(host_ctl);
        host_ctl = nullptr;
        host_bytes = 0;
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (cap_stream) cudaStreamDestroy(cap_stream);
        if (up) cudaStreamDestroy(up);
        up = nullptr;
        if (uploaded) cudaEventDestroy(uploaded);
        uploaded = nullptr;
        for (auto &x : side)
            if (x) cudaStreamDestroy(x);
        for (auto &x : join)
            if (x) cudaEventDestroy(x);
        if (fork) cudaEventDestroy(fork);
        exec = nullptr;
        graph = nullptr;
        cap_stream = nullptr;
        for (auto &x : side) x = nullptr;
        for (auto &x : join) x = nullptr;
        fork = nullptr;
    }
};

namespace {

// (Re)build batch b for these jobs: per-circuit arguments and prefixes in
// one device block, which is reused when it is large enough.
// up: the stream that uploads the control block, in order before the next
// pass on it (the caller then must not rebind or destroy the batch before
// that pass is done); null: uploaded on a stream of the batch's own, which
// the next pass waits for on the device.
pdf_status batch_build(pdf_batch *b, const pdf_batch_job *jobs, uint32_t n_jobs, uint32_t flags,
                       cudaStream_t up = nullptr) {
    if (!jobs || !n_jobs || (flags & ~(uint32_t)(PDF_BATCH_APPEND | PDF_BATCH_NO_GRAPH))) return PDF_EINVAL;
    pdf_circuit *c0 = jobs[0].circuit;
    if (!c0) return PDF_EINVAL;
    for (uint32_t i = 0; i < n_jobs; i++) {
        const pdf_batch_job &j = jobs[i];
        if (!j.circuit || !j.state || j.state->c != j.circuit || j.circuit->device != c0->device ||
            j.circuit->mark_mode != c0->mark_mode)
            return PDF_EINVAL;
        if (j.circuit->seg_len > 1) return PDF_ENOTSUP;  // batches grade segments of one net
        const uint64_t n = j.pairs.n_pairs, W = (n + 31) / 32;
        if (n == 0 || !j.pairs.on_device || j.pair_base + n > 0xFFFFFFFFull ||
            !planes_fit(j.circuit, W, j.pairs.ld, {j.pairs.v, j.pairs.t}))
            return PDF_EINVAL;
    }
    b->drop_graph();
    b->ran = false;
    // blocks that only the binding before this one held may be freed from here on
    b->bound = std::make_shared<char>();
    b->device = c0->device;
    b->circuits.clear();
    b->states.clear();
    b->gate_evals = 0;
    std::vector<FwdArgs> fa(n_jobs);
    std::vector<CoverArgs> ca(n_jobs);
    std::vector<uint32_t> bp(n_jobs + 1, 0), gp(n_jobs + 1, 0);
    uint64_t items = 0;
    BatchLaunch &L = b->L;
    L = BatchLaunch{};
    L.sem = (uint32_t)c0->mark_mode;
    L.hash_cap = c0->hash_cap;
    // Jobs in classes of equal tile width and CTAs per SM (1, 2, 4), each
    // class one forward launch (its kernel, block size and shared memory
    // sized for its members), so the CTAs of narrow circuits share SMs
    // instead of holding the shared memory of the widest member; within a
    // class the longest CTA walks go first.
    std::vector<Walk> walks(n_jobs);
    uint64_t res_ctas = 0, lane_ctas = 0, all_words = 0;
    double rounds = 0;  // of blocks of the netlists that fit on chip only just
    for (uint32_t i = 0; i < n_jobs; i++) {
        const Plan &p = jobs[i].circuit->lean();
        const uint64_t W = (jobs[i].pairs.n_pairs + 31) / 32;
        all_words += W;
        if (p.image) {
            const uint32_t at_once = resident_shape(p.res, W).words;
            if (at_once < kResidentWords) rounds += (double)W / (at_once * p.res.sms);
        } else if (p.wide) {
            lane_ctas += (W + p.bw - 1) / p.bw;
        }
    }
    const uint64_t sms = c0->full.res.sms;
    const bool lanes = lane_ctas >= batch_lanes_from(sms);
    // (as resident_pays, over all the jobs)
    const bool chip = rounds <= 2.5 * std::max(1.0, (double)all_words / (10.0 * sms));
    for (uint32_t i = 0; i < n_jobs; i++) {
        const uint64_t W = (jobs[i].pairs.n_pairs + 31) / 32;
        const Plan &p = jobs[i].circuit->lean();
        Walk &k = walks[i] = jobs[i].circuit->batch_walk(
            W, lanes, chip || (p.image && resident_shape(p.res, W).words >= kResidentWords));
        if (!k.resident) continue;
        // a CTA takes blocks worth about twice its copy of the image
        const double load = 2.0 + k.p->res.image_bytes / 95e3;
        k.rs.per = std::min(k.rs.blocks, 1 + (uint32_t)(2 * load / (k.rs.block_us * k.rs.occ)));
        res_ctas += (k.rs.blocks + k.rs.per - 1) / k.rs.per;
    }
    // ... or fewer while that leaves SMs without a CTA
    for (Walk &k : walks)
        if (k.resident && res_ctas < 2 * sms)
            k.rs.per = std::max<uint32_t>(1, (uint32_t)(k.rs.per * res_ctas / (2 * sms)));
    // Jobs of one block width whose CTAs all fit the GPU at the lowest occupancy
    // among them share one launch.
    for (uint32_t bw = 1; bw <= 8; bw *= 2) {
        uint64_t ctas = 0;
        uint32_t low = ~0u;
        for (const Walk &k : walks)
            if (k.resident && k.bw == bw) {
                ctas += (k.rs.blocks + k.rs.per - 1) / k.rs.per;
                low = std::min(low, k.rs.occ);
            }
        if (ctas && ctas <= sms * low)
            for (Walk &k : walks)
                if (k.resident && k.bw == bw) k.rs.occ = low;
    }
    const auto occ = [](const Walk &k) { return k.resident ? k.rs.occ : k.p->occ; };
    std::vector<uint32_t> order(n_jobs);
    for (uint32_t i = 0; i < n_jobs; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
        const Walk &kx = walks[x], &ky = walks[y];
        if (kx.resident != ky.resident) return ky.resident;
        if (kx.bw != ky.bw) return kx.bw > ky.bw;
        if (occ(kx) != occ(ky)) return occ(kx) < occ(ky);
        if (kx.resident) return kx.rs.per * kx.rs.block_us > ky.rs.per * ky.rs.block_us;
        return kx.p->chain > ky.p->chain;
    });
    for (uint32_t k = 0; k < n_jobs; k++) {
        const pdf_batch_job &j = jobs[order[k]];
        const uint32_t i = k;
        pdf_circuit *c = j.circuit;
        pdf_state *s = j.state;
        const Walk &wk = walks[order[k]];
        const Plan &p = *wk.p;
        const uint64_t n = j.pairs.n_pairs, W = (n + 31) / 32, G = p.n_gates;
        if (ensure_ws(c, wk, s->ws, W, true) != PDF_OK) return PDF_ENOMEM;
        if (!s->ws.hold_for(b->bound)) return PDF_ENOMEM;  // the batch's arguments hold its addresses
        FwdArgs a = base_fwd(c, wk, n);
        a.pi_v = j.pairs.v;
        a.pi_t = j.pairs.t;
        a.pi_ld = j.pairs.ld;
        a.store_all = 0;
        a.in_pieces = p.in_pieces;
        use_ws_planes(a, wk, s->ws, W);
        const Scratch x = ws_scratch(c, wk, s->ws, W);
        use_scratch(a, x);
        a.first_x = s->first_x.as<uint32_t>();
        a.first_y = s->first_y.as<uint32_t>();
        a.pair_base = (uint32_t)j.pair_base;
        DevAcc *acc = s->acc.as<DevAcc>();
        a.err = &acc->err;
        a.acc = acc;
        a.active = x.active;
        fa[i] = a;
        ca[i] = base_cover(c, wk, s->ws, a.M, a.ld, n, (uint32_t)j.pair_base, a.first_x, a.first_y, acc);
        ca[i].mirror = s->mirror;
        const uint64_t blocks = wk.resident ? (wk.rs.blocks + wk.rs.per - 1) / wk.rs.per : (W + p.bw - 1) / p.bw;
        if (bp[i] + blocks > 0x7FFFFFFFull || gp[i] + G > 0xFFFFFFFFull) return PDF_ENOTSUP;
        bp[i + 1] = bp[i] + (uint32_t)blocks;
        gp[i + 1] = gp[i] + (uint32_t)G;
        items += std::min<uint64_t>(W * 32, 2 * G);
        L.tile = std::max(L.tile, c->bw);
        L.threads = std::max(L.threads, c->full.threads);
        const size_t smem = wk.resident ? wk.rs.smem : p.fwd_smem;
        L.fwd_smem = std::max(L.fwd_smem, smem);
        L.cover_grid = std::max(L.cover_grid, c->cover_grid);
        if (!L.n_class || L.cls[L.n_class - 1].occ != occ(wk) || L.cls[L.n_class - 1].bw != wk.bw ||
            L.cls[L.n_class - 1].resident != (wk.resident ? 1u : 0u)) {
            if (L.n_class == kMaxBatchClasses) return PDF_ENOTSUP;
            BatchClass &k2 = L.cls[L.n_class++];
            k2.bw = wk.bw;
            k2.occ = occ(wk);
            k2.resident = wk.resident ? 1u : 0u;
            k2.blk0 = bp[i];
        }
        BatchClass &cl = L.cls[L.n_class - 1];
        cl.threads = std::max(cl.threads, wk.resident ? wk.rs.threads : p.threads);
        cl.smem = std::max(cl.smem, smem);
        b->gate_evals += (uint64_t)c->info.n_gates * n;
        b->circuits.push_back(c);
        b->states.push_back(s);
    }
    // one side stream and join event per class after the first
    if (!b->fork) PDF_CUDA(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
    for (uint32_t k = 1; k < L.n_class; k++) {
        if (!b->side[k - 1]) PDF_CUDA(cudaStreamCreateWithFlags(&b->side[k - 1], cudaStreamNonBlocking));
        if (!b->join[k - 1]) PDF_CUDA(cudaEventCreateWithFlags(&b->join[k - 1], cudaEventDisableTiming));
    }
    for (uint32_t k = 0; k + 1 < kMaxBatchClasses; k++) {
        L.side[k] = b->side[k];
        L.join[k] = b->join[k];
    }
    L.fork = b->fork;
    b->use_graph = !(flags & PDF_BATCH_NO_GRAPH);
    // inside a captured graph the events are external nodes; run directly, plain records
    for (uint32_t k = 0; k < 3; k++) L.prof[k] = b->profiling ? b->prof[k] : nullptr;
    L.prof_external = b->use_graph ? 1u : 0u;
    L.n = n_jobs;
    L.total_blocks = bp[n_jobs];
    for (uint32_t k = 0; k < L.n_class; k++)
        L.cls[k].blocks = (k + 1 < L.n_class ? L.cls[k + 1].blk0 : L.total_blocks) - L.cls[k].blk0;
    L.total_gates = gp[n_jobs];
    L.append = (flags & PDF_BATCH_APPEND) ? 1u : 0u;
    // the small-table cover that runs first (several CTAs per SM)
    if (!b->small_cap) {  // once per batch (its device does not change)
        b->small_cap = cover_small_cap(b->device, &b->small_per_sm);
        if (!b->small_cap) return PDF_ECUDA;
    }
    L.small_cap = std::min(b->small_cap, L.hash_cap);
    L.small_grid = L.cover_grid * b->small_per_sm;
    // one device block: control word, circuit arguments, prefixes, then the
    // item lists (all items; those passed to the large table; those queued
    // for the spill cover)
    auto a256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t list = a256(sizeof(uint2) * std::max<uint64_t>(items, 1));
    const size_t o_f = a256(sizeof(BatchCtl)), o_c = o_f + a256(sizeof(FwdArgs) * n_jobs),
                 o_b = o_c + a256(sizeof(CoverArgs) * n_jobs), o_g = o_b + a256(4 * (n_jobs + 1)),
                 o_i = o_g + a256(4 * (n_jobs + 1)), o_m = o_i + list, o_o = o_m + list, total = o_o + list;
    // the spill cover: as many CTAs as the spilling circuit with the fewest
    // slots has (circuits without slots cannot spill)
    L.spill_grid = 0;
    for (uint32_t i = 0; i < n_jobs; i++)
        if (ca[i].spill_slots) L.spill_grid = L.spill_grid ? std::min(L.spill_grid, ca[i].spill_slots) : ca[i].spill_slots;
    // The block is written into mapped pinned host memory and pulled to the
    // device by a small kernel on the batch's own stream: a copy-engine
    // transfer would queue behind other host threads' bulk uploads (a
    // server's arriving jobs), which held passes up for hundreds of ms.
    if (b->host_bytes < o_i) {
        if (b->uploaded) PDF_CUDA(cudaEventSynchronize(b->uploaded));
        const size_t want = std::max<size_t>({o_i, 2 * b->host_bytes, (size_t)256 << 10});
        if (b->host_ctl) cudaFreeHost(b->host_ctl);
        b->host_ctl = nullptr;
        b->host_bytes = 0;
        if (cudaHostAlloc(reinterpret_cast<void **>(&b->host_ctl), want, cudaHostAllocMapped) != cudaSuccess)
            return PDF_ENOMEM;
        b->host_bytes = want;
    }
    // (the upload before this one may not have been run, or waited for, yet)
    if (b->uploaded) PDF_CUDA(cudaEventSynchronize(b->uploaded));
    unsigned char *hbuf = b->host_ctl;
    std::memset(hbuf, 0, o_i);
    std::memcpy(hbuf + o_f, fa.data(), sizeof(FwdArgs) * n_jobs);
    std::memcpy(hbuf + o_c, ca.data(), sizeof(CoverArgs) * n_jobs);
    std::memcpy(hbuf + o_b, bp.data(), 4 * (n_jobs + 1));
    std::memcpy(hbuf + o_g, gp.data(), 4 * (n_jobs + 1));
    // grown geometrically: freeing the old block waits for the whole device
    if (total > b->ctl.bytes && b->ctl.ensure(std::max<size_t>({total, 2 * b->ctl.bytes, (size_t)1 << 20})) != cudaSuccess)
        return PDF_ENOMEM;
    void *src = nullptr;
    if (!up && !b->up) PDF_CUDA(cudaStreamCreateWithFlags(&b->up, cudaStreamNonBlocking));
    if (!up && !b->uploaded) PDF_CUDA(cudaEventCreateWithFlags(&b->uploaded, cudaEventDisableTiming));
    PDF_CUDA(cudaHostGetDevicePointer(&src, hbuf, 0));
    L.host_ctl = static_cast<BatchCtl *>(src);
    // the launch below is checked with cudaGetLastError, which would also
    // report an unchecked failure left on this thread by an earlier call
    // (this library's or the caller's); start from a clean slate
    (void)cudaGetLastError();
    PDF_CUDA(launch_copy_from_host(b->ctl.p, src, o_i / 16, up ? up : b->up));
    b->wait_upload = !up;
    if (!up) PDF_CUDA(cudaEventRecord(b->uploaded, b->up));
    unsigned char *base = b->ctl.as<unsigned char>();
    L.ctl = reinterpret_cast<BatchCtl *>(base);
    L.fargs = reinterpret_cast<FwdArgs *>(base + o_f);
    L.cargs = reinterpret_cast<CoverArgs *>(base + o_c);
    L.bpref = reinterpret_cast<const uint32_t *>(base + o_b);
    L.gpref = reinterpret_cast<const uint32_t *>(base + o_g);
    L.items = reinterpret_cast<uint2 *>(base + o_i);
    L.mid_items = reinterpret_cast<uint2 *>(base + o_m);
    L.over_items = reinterpret_cast<uint2 *>(base + o_o);
    b->bytes = b->ctl.bytes;
    PDF_CUDA(prepare_batch(L));
    if (b->use_graph && !b->cap_stream &&
        cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking) != cudaSuccess)
        return PDF_ECUDA;
    return PDF_OK;
}

}  // namespace

extern "C" pdf_status pdf_batch_create(const pdf_batch_job *jobs, uint32_t n_jobs, uint32_t flags, pdf_batch **out) {
    if (!out) return PDF_EINVAL;
    *out = nullptr;
    if (!jobs || !n_jobs || !jobs[0].circuit) return PDF_EINVAL;
    DeviceGuard dg(jobs[0].circuit->device);
    if (!dg.ok) return PDF_ECUDA;
    pdf_batch *b = new (std::nothrow) pdf_batch();
    if (!b) return PDF_ENOMEM;
    const pdf_status st = batch_build(b, jobs, n_jobs, flags);
    if (st != PDF_OK) {
        b->release();
        delete b;
        (void)cudaGetLastError();
        return st;
    }
    *out = b;
    return PDF_OK;
}

extern "C" pdf_status pdf_batch_rebind(pdf_batch *b, const pdf_batch_job *jobs, uint32_t n_jobs, uint32_t flags) {
    if (!b || !jobs || !n_jobs || !jobs[0].circuit || jobs[0].circuit->device != b->device) return PDF_EINVAL;
    DeviceGuard dg(b->device);
    if (!dg.ok) return PDF_ECUDA;
    const pdf_status st = batch_build(b, jobs, n_jobs, flags);
    if (st != PDF_OK) (void)cudaGetLastError();
    return st;
}

extern "C" void pdf_batch_destroy(pdf_batch *b) {
    if (!b) return;
    DeviceGuard dg(b->device);
    b->release();
    delete b;
}

extern "C" pdf_status pdf_batch_query(const pdf_batch *b, pdf_batch_info *info) {
    if (!b || !info) return PDF_EINVAL;
    info->n_jobs = b->L.n;
    info->tile_words = b->L.tile;  // the widest circuit tile
    info->threads = b->L.threads;
    info->ctas = b->L.total_blocks;
    info->gate_evals = b->gate_evals;
    info->device_bytes = b->bytes;
    info->forward_launches = 0;
    for (uint32_t k = 0; k < b->L.n_class; k++) info->forward_launches += b->L.cls[k].blocks ? 1u : 0u;
    info->launches = info->forward_launches + (b->L.spill_grid ? 4 : 3);
    return PDF_OK;
}

extern "C" pdf_status pdf_batch_run_async(pdf_batch *b, void *stream) {
    if (!b) return PDF_EINVAL;
    DeviceGuard dg(b->device);
    if (!dg.ok) return PDF_ECUDA;
    (void)cudaGetLastError();  // an unchecked failure of an earlier call is not this run's
    if (b->wait_upload) {
        // in stream order; a stream that the caller captures cannot wait for
        // work outside its graph, so there the host does
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        PDF_CUDA(cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &cap));
        if (cap != cudaStreamCaptureStatusNone) PDF_CUDA(cudaEventSynchronize(b->uploaded));
        else PDF_CUDA(cudaStreamWaitEvent(static_cast<cudaStream_t>(stream), b->uploaded, 0));
        b->wait_upload = false;
    }
    // A graph pays from its second replay on (capturing, instantiating and
    // destroying one takes over 200 us, more than a small pass): a batch that is
    // bound anew for every pass launches directly.
    if (!b->use_graph || (!b->exec && !b->ran)) {
        BatchLaunch L = b->L;
        L.prof_external = 0;
        PDF_CUDA(launch_batch(L, static_cast<cudaStream_t>(stream)));
        b->ran = true;
        return PDF_OK;
    }
    if (!b->exec) {  // capture the launches once
        PDF_CUDA(cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeThreadLocal));
        const cudaError_t le = launch_batch(b->L, b->cap_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(b->cap_stream, &g);
        if (le != cudaSuccess || ce != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            (void)cudaGetLastError();
            return PDF_ECUDA;
        }
        b->graph = g;
        PDF_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
    }
    PDF_CUDA(cudaGraphLaunch(b->exec, static_cast<cudaStream_t>(stream)));
    return PDF_OK;
}

extern "C" pdf_status pdf_batch_profile(pdf_batch *b, int enable) {
    if (!b) return PDF_EINVAL;
    DeviceGuard dg(b->device);
    if (!dg.ok) return PDF_ECUDA;
    if (enable && !b->prof[0])
        for (auto &e : b->prof) PDF_CUDA(cudaEventCreate(&e));
    b->profiling = enable != 0;
    for (uint32_t k = 0; k < 3; k++) b->L.prof[k] = b->profiling ? b->prof[k] : nullptr;
    b->drop_graph();  // captured again at the next run, with or without the events
    return PDF_OK;
}

extern "C" pdf_status pdf_batch_profile_read(pdf_batch *b, double *ms) {
    if (!b || !ms || !b->profiling) return PDF_EINVAL;
    DeviceGuard dg(b->device);
    if (!dg.ok) return PDF_ECUDA;
    float f = 0.0f, c = 0.0f;
    PDF_CUDA(cudaEventSynchronize(b->prof[2]));
    PDF_CUDA(cudaEventElapsedTime(&f, b->prof[0], b->prof[1]));
    PDF_CUDA(cudaEventElapsedTime(&c, b->prof[1], b->prof[2]));
    ms[0] = f;
    ms[1] = c;
    return PDF_OK;
}

pdf_status batch_rebind_on(pdf_batch *b, const pdf_batch_job *jobs, uint32_t n_jobs, uint32_t flags,
                           cudaStream_t stream) {
    if (!b || !jobs || !n_jobs || !jobs[0].circuit || jobs[0].circuit->device != b->device || !stream)
        return PDF_EINVAL;
    DeviceGuard dg(b->device);
    if (!dg.ok) return PDF_ECUDA;
    const pdf_status st = batch_build(b, jobs, n_jobs, flags, stream);
    if (st != PDF_OK) (void)cudaGetLastError();
    return st;
}

pdf_status batch_pass_async(pdf_batch *b, cudaStream_t stream) {
    return pdf_batch_run_async(b, stream);
}

pdf_status batch_pass_status(const pdf_batch *b) {
    return err_status(reinterpret_cast<const BatchCtl *>(b->host_ctl)->err);
}

extern "C" pdf_status pdf_batch_run(pdf_batch *b, void *stream) {
    pdf_status st = pdf_batch_run_async(b, stream);
    if (st != PDF_OK) return st;
    DeviceGuard dg(b->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    PDF_CUDA(cudaStreamSynchronize(cs));
    return batch_pass_status(b);  // the control word, left there by the kernel that closed the pass
}

// Autotuner of the batch tile width: times the whole batch at each candidate.
extern "C" pdf_status pdf_batch_autotune(const pdf_netlist *const *netlists, const uint64_t *n_pairs, uint32_t n,
                                         const pdf_circuit_opts *base, uint32_t reps, pdf_circuit_opts *best,
                                         float *best_ms) {
    if (!netlists || !n_pairs || !n || !best || reps == 0) return PDF_EINVAL;
    const pdf_circuit_opts b0 = base ? *base : pdf_circuit_opts{};
    DeviceGuard dg(b0.device);
    if (!dg.ok) return PDF_ECUDA;
    float best_t = 0.0f;
    uint32_t best_w = 0, best_threads = 0;
    pdf_status last = PDF_OK;
    // candidates: tile width x block size (the default, piece capacity + 64,
    // or 256 threads: pieces of 192 gates and more CTAs per SM), unless the
    // caller fixed the block size
    std::vector<std::pair<uint32_t, uint32_t>> cand;
    for (uint32_t tw : {2u, 4u, 8u})
        for (uint32_t th : {0u, 256u})
            if (!b0.threads || th == 0) cand.push_back({tw, b0.threads ? b0.threads : th});
    if (!b0.threads) {  // the lane tiles
        cand.push_back({kLaneWords, 0u});
        cand.push_back({kLaneWords2, 0u});
        cand.push_back({kLaneWords4, 0u});
    }
    for (const auto &cw : cand) {
        const uint32_t tw = cw.first;
        pdf_circuit_opts o = b0;
        o.tile_words = tw;
        o.threads = cw.second;
        std::vector<pdf_circuit *> cs(n, nullptr);
        std::vector<pdf_state *> ss(n, nullptr);
        std::vector<void *> bufs(n, nullptr);
        std::vector<pdf_batch_job> jobs(n);
        pdf_batch *b = nullptr;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        pdf_status st = PDF_OK;
        for (uint32_t i = 0; i < n && st == PDF_OK; i++) {
            st = pdf_circuit_create(netlists[i], &o, &cs[i]);
            if (st == PDF_OK) st = pdf_state_create(cs[i], &ss[i]);
            if (st != PDF_OK) break;
            const uint64_t np = n_pairs[i], W = (np + 31) / 32, ld = (W + tw - 1) / tw * tw;
            const uint32_t npi = cs[i]->info.n_pi;
            std::vector<uint32_t> v(npi * ld), t(npi * ld);
            st = pdf_gen_pairs(0x7A11u + i, npi, np, ld, v.data(), t.data());
            if (st != PDF_OK) break;
            if (cudaMalloc(&bufs[i], 2 * npi * ld * 4) != cudaSuccess) {
                st = PDF_ENOMEM;
                break;
            }
            uint32_t *dv = static_cast<uint32_t *>(bufs[i]), *dt = dv + npi * ld;
            if (cudaMemcpy(dv, v.data(), npi * ld * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
                cudaMemcpy(dt, t.data(), npi * ld * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
                st = PDF_ECUDA;
                break;
            }
            jobs[i] = pdf_batch_job{cs[i], ss[i], pdf_pairs{dv, dt, np, ld, 1}, 0};
        }
        if (st == PDF_OK) st = pdf_batch_create(jobs.data(), n, 0, &b);
        for (int r = 0; r < 2 && st == PDF_OK; r++) st = pdf_batch_run(b, nullptr);  // warm-up; the second captures the graph
        float ms = 0.0f;
        if (st == PDF_OK) {
            if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess ||
                cudaEventRecord(e0, nullptr) != cudaSuccess)
                st = PDF_ECUDA;
            for (uint32_t r = 0; r < reps && st == PDF_OK; r++) st = pdf_batch_run_async(b, nullptr);
            if (st == PDF_OK && (cudaEventRecord(e1, nullptr) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                                 cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
                st = PDF_ECUDA;
        }
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        pdf_batch_destroy(b);
        for (uint32_t i = 0; i < n; i++) {
            pdf_state_destroy(ss[i]);
            pdf_circuit_destroy(cs[i]);
            if (bufs[i]) cudaFree(bufs[i]);
        }
        (void)cudaGetLastError();
        if (st != PDF_OK) {  // a tile that does not fit is skipped
            last = st;
            continue;
        }
        ms /= (float)reps;
        if (!best_w || ms < best_t) {
            best_t = ms;
            best_w = tw;
            best_threads = cw.second;
        }
    }
    if (!best_w) return last;
    *best = b0;
    best->tile_words = best_w;
    best->threads = best_threads;
    if (best_ms) *best_ms = best_t;
    return PDF_OK;
}

// One sizing for all the walks: growing a block step by step would free each
// step's, and cudaFree waits for the whole device.
extern "C" pdf_status pdf_state_reserve(pdf_state *s, uint64_t n_pairs) {
    if (!s || !n_pairs) return PDF_EINVAL;
    DeviceGuard dg(s->c->device);
    if (!dg.ok) return PDF_ECUDA;
    std::lock_guard<std::mutex> lk(s->mu);
    const uint64_t W = (n_pairs + 31) / 32;
    pdf_circuit *c = s->c;
    WsNeed need;
    need.lean(c, c->lean_walk(W), W);
    if (c->seg_len <= 1) need.batch(c, W);
    need.out(c, c->planes_walk(W), W, RES_PLANES, true).with(c, c->full_walk(W), W, !c->out_plan);
    return ensure_ws(c, need, s->ws, W);
}

// The workspace of a state that only batches grade.
pdf_status state_reserve_batch(pdf_state *s, uint64_t n_pairs) {
    DeviceGuard dg(s->c->device);
    if (!dg.ok) return PDF_ECUDA;
    std::lock_guard<std::mutex> lk(s->mu);
    const uint64_t W = (n_pairs + 31) / 32;
    return ensure_ws(s->c, WsNeed{}.batch(s->c, W), s->ws, W);
}
