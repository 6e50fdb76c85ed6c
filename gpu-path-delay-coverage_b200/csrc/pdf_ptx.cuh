// pdf_ptx.cuh -- device helpers shared by the kernel files.
#ifndef PDF_PTX_CUH
#define PDF_PTX_CUH

#include "pdf_kernels.cuh"

namespace {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;

// The caller's id of gate g of a (possibly reduced) netlist, kEmpty for a
// constant: the index of its first-detect ids.
__device__ __forceinline__ uint32_t net_id(const DevCircuit &c, uint32_t g) { return c.orig ? __ldg(c.orig + g) : g; }

__device__ __forceinline__ GateRec load_rec(const GateRec *p) {
    const uint4 *q = reinterpret_cast<const uint4 *>(p);
    const uint4 a = __ldg(q), b = __ldg(q + 1);
    GateRec r;
    r.w[0] = a.x;
    r.w[1] = a.y;
    r.w[2] = a.z;
    r.w[3] = a.w;
    r.w[4] = b.x;
    r.w[5] = b.y;
    r.w[6] = b.z;
    r.w[7] = b.w;
    return r;
}

__device__ __forceinline__ bool bit_test(const uint32_t *bm, uint32_t g) { return (bm[g >> 5] >> (g & 31)) & 1u; }

// ---- TMA bulk copies and mbarriers (inline PTX, sm_90+ / sm_100a) ----

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *m, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *m, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes)
                 : "memory");
}
// One untiled bulk copy global -> shared; both addresses 16-byte aligned,
// bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *m) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(m))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *m, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(phase)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t *m, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(phase)
        : "memory");
    return ok != 0;
}
// Every wait is bounded: on expiry the caller reports PDF_ETIMEOUT.  polls =
// 0: up to kSpinLimit blocking polls (try_wait may suspend the thread until
// the phase completes); polls > 0: that many non-blocking polls, a bound
// small enough to run out (tests of the timeout path).
constexpr uint32_t kSpinLimit = 1u << 24;
__device__ __forceinline__ bool mbar_wait(uint64_t *m, uint32_t phase, uint32_t polls = 0) {
    if (polls) {
        for (uint32_t i = 0; i < polls; i++)
            if (mbar_test_wait(m, phase)) return true;
        return false;
    }
    for (uint32_t i = 0; i < kSpinLimit; i++)
        if (mbar_try_wait(m, phase)) return true;
    return false;
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Launches of one call follow each other without the gap between grids (about
// 1.5 us each): the next one is started once every CTA of this one has passed
// grid_trigger, and waits in grid_wait until this one is complete and visible.
// Each kernel launched by launch_next waits before it ends, so that whatever
// follows it in the stream follows all before it too.
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
cudaError_t launch_next(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchConfig_t c{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Last i with pref[i] <= x.
__device__ __forceinline__ uint32_t prefix_find(const uint32_t *pref, uint32_t n, uint32_t x) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(pref + mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The first forward CTA of a pass clears the batch's control word.
__device__ __forceinline__ void batch_begin(BatchCtl *ctl) {
    ctl->n_items = 0;
    ctl->done = 0;
    ctl->err = 0;
    ctl->n_over = 0;
    ctl->done_over = 0;
    ctl->n_mid = 0;
    ctl->done_mid = 0;
}

}  // namespace

#endif
