// Thin wrappers over the sm_90+/sm_100a PTX used by the pipelined kernels:
// mbarriers, TMA tensor loads (no multicast), and a bounded mbarrier wait.
#pragma once

#include <cstdint>

#include <cuda.h>
#include <cuda_runtime.h>

namespace lk::ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

// Makes mbarrier initialisation visible to the async proxy (TMA).
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// To be called before a stage of a copy ring is released, with z formed from a
// value of every load from it: an arrival does not wait for the results of loads
// issued before it (a warp or proxy fence between them does not either), and the
// copy that refills the stage can overtake them. Seen in the sample-walking folds
// with few warps a block and several blocks an SM: rows of a word held the samples
// of the word that replaced it. Testing z makes the arrival, which follows in
// program order, issue after the values have been read; the branch only tests the
// barrier again. It costs those folds 1 to 4 %.
__device__ __forceinline__ void loads_done(uint32_t z, uint64_t* bar, uint32_t parity) {
    if (z == 0x9e3779b9u) {
        mbar_try_wait(bar, parity);
    }
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Every device-side wait is bounded: at most kWaitLimitNs of wall time (read
// from %globaltimer every 256 polls) and at most kSpinLimit polls. On expiry
// the caller records a status bit and returns instead of spinning forever.
constexpr uint64_t kWaitLimitNs = 500000000ull;  // 0.5 s
constexpr uint32_t kSpinLimit = 1u << 20;

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  uint32_t* status, uint32_t bit,
                                                  uint64_t limit_ns = kWaitLimitNs) {
    if (mbar_try_wait(bar, parity)) {
        return true;
    }
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 1; it < kSpinLimit; ++it) {
        if (mbar_try_wait(bar, parity)) {
            return true;
        }
        if ((it & 255u) == 0 && globaltimer_ns() - t0 > limit_ns) {
            break;
        }
    }
    atomicOr(status, bit);
    return false;
}

// 3-D tiled TMA load global -> shared, completion signalled on `bar`.
// Plain (no multicast) form; the destination is this CTA's shared memory.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// Untiled bulk copy global -> shared (16-byte aligned addresses and size, no
// multicast), completion signalled on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// 2-D tiled TMA load global -> shared (no multicast).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}

// ---- tensor memory (tcgen05, sm_100a) -----------------------------------
// Allocation of ncols columns (a power of two in [32, 512]) for the CTA by
// one whole warp; the TMEM address is written to *dst (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Thread t of the warp writes (a, b) to columns col, col + 1 of its lane
// (the warp's 32-lane quadrant is in the address's lane field).
__device__ __forceinline__ void tmem_st2(uint32_t taddr, float a, float b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "f"(a), "f"(b)
                 : "memory");
}
// Asynchronous read of two columns; the values are valid after tmem_wait_ld.
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, float& a, float& b) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(taddr)
                 : "memory");
}
// Waits for this thread's TMEM reads; the named registers are tied to the
// wait so no use of them is scheduled before it.
__device__ __forceinline__ void tmem_wait_ld(float& a, float& b) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(a), "+f"(b)::"memory");
}
__device__ __forceinline__ void tmem_wait_ld4(float4& a, float4& b) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w), "+f"(b.x), "+f"(b.y), "+f"(b.z), "+f"(b.w)::"memory");
}
__device__ __forceinline__ void tmem_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

}  // namespace lk::ptx
