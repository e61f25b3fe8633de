// Thin wrappers over the sm_100a instructions that the tensor-core kernels use:
// mbarriers with bounded waits, TMA tiled loads (never multicast), tensor
// memory allocation, tcgen05.mma / commit / ld, and the shared-memory and
// instruction descriptors of tcgen05.  Layouts of the descriptors follow the
// public PTX documentation of the tcgen05 family.
#pragma once

#include <cuda.h>  // CUtensorMap (types only; the driver is reached through cudaGetDriverEntryPoint)

#include "common.cuh"

namespace sm100 {

__device__ __forceinline__ uint32_t smem_addr(const void* ptr) { return (uint32_t)__cvta_generic_to_shared(ptr); }

__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(pred));
    return pred != 0;
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Waits for the phase with the given parity.  The wait is bounded: after
// `limit` polls it gives up and returns false, and the caller records the
// failure and winds the kernel down instead of hanging the device.
#define KIRAI_WAIT_LIMIT (1u << 24)
__device__ __forceinline__ bool mbar_wait_limited(uint32_t bar, uint32_t parity, uint32_t limit) {
    for (uint32_t spin = 0; spin < limit; ++spin) {
        if (mbar_test(bar, parity)) return true;
        if (spin > 64) __nanosleep(spin > 4096 ? 256 : 32);
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) { return mbar_wait_limited(bar, parity, KIRAI_WAIT_LIMIT); }

// The same for waits on the critical path of a pipeline (between an MMA and the warps that consume
// its result): polls without sleeping for a long while, so that the wake-up adds no latency.
__device__ __forceinline__ bool mbar_wait_hot(uint32_t bar, uint32_t parity) {
    for (uint32_t spin = 0; spin < KIRAI_WAIT_LIMIT; ++spin) {
        if (mbar_test(bar, parity)) return true;
        if (spin > (1u << 16)) __nanosleep(64);
    }
    return false;
}

// ----------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_descriptor(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
// 2-D tiled load of one box into shared memory; x is the innermost (contiguous)
// coordinate in elements and must make x * element size a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// Untiled bulk copy of `bytes` contiguous bytes into shared memory (both addresses 16-byte aligned, the size a
// multiple of 16), counted on the barrier like a tiled load.
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

// The same for bytes that are read once: they are the first to leave L2 again.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}
__device__ __forceinline__ void bulk_load_1d_once(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t evict_first) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar), "l"(evict_first)
                 : "memory");
}

// ------------------------------------------------------------- tensor memory
// `tmem_alloc` waits until the columns are free, without a limit, and a kernel may hold columns while it waits for the kernels
// ahead of it in its stream.  So that no two of them wait for each other:
//  * a kernel that takes its columns after pdl_wait() lets the next kernel start only once it has them: a CTA of the next one
//    that came first would keep the columns and wait for the end of this one, which would wait for the columns;
//  * a CTA that takes all 512 columns asks for at least ALL_COLUMNS_SHARED bytes of shared memory, beside which no other CTA that
//    uses tensor memory fits an SM (`alone_with_all_columns`, asserted by each of these kernels with its smallest size).
// The other kernels take their columns ahead of pdl_wait(), and those of any of their CTAs that fit an SM together are at most 512
// (32 columns with 75 KB, 64 and 128 with 99, 256 with 83 or 195).
constexpr int SM_SHARED = 228 * 1024, CTA_SHARED_RESERVED = 1024;  // bytes of an SM, and what the system takes for each of its CTAs
constexpr int ALL_COLUMNS_SHARED = 192 * 1024;
constexpr bool alone_with_all_columns(int dynamic_bytes) {
    return dynamic_bytes + CTA_SHARED_RESERVED + ALL_COLUMNS_SHARED + CTA_SHARED_RESERVED > SM_SHARED;
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t columns) {  // whole warp; columns: power of 2 >= 32
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(columns) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {  // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory operand descriptor for a K-major tile whose rows are 128 bytes
// (64 bf16) and which TMA wrote with the 128-byte swizzle: 8-row groups are
// 1024 bytes apart (stride byte offset), the leading offset is unused (1), the
// descriptor version is 1 and the layout type 2 (SWIZZLE_128B).
// The same with the 8-row groups `group_bytes` apart (tiles whose groups interleave several 64-column panels).
__device__ __forceinline__ uint64_t smem_desc_k_major_sw128_groups(uint32_t addr, uint32_t group_bytes) {
    uint64_t desc = 0;
    desc |= (uint64_t)((addr & 0x3FFFF) >> 4);
    desc |= (uint64_t)1 << 16;
    desc |= (uint64_t)((group_bytes >> 4) & 0x3FFF) << 32;
    desc |= (uint64_t)1 << 46;
    desc |= (uint64_t)2 << 61;
    return desc;
}
__device__ __forceinline__ uint64_t smem_desc_k_major_sw128(uint32_t addr) {
    uint64_t desc = 0;
    desc |= (uint64_t)((addr & 0x3FFFF) >> 4);
    desc |= (uint64_t)1 << 16;
    desc |= (uint64_t)(1024 >> 4) << 32;
    desc |= (uint64_t)1 << 46;
    desc |= (uint64_t)2 << 61;
    return desc;
}

// Instruction descriptor of tcgen05.mma.kind::f16 with bf16 operands (both
// K-major), 32-bit accumulation, an M x N tile.
__host__ __device__ constexpr uint32_t instr_desc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread.
__device__ __forceinline__ void mma_bf16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier when every MMA issued so far by this thread is done.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ------------------------------------------------------------------ clusters
// Shared memory of another CTA of the cluster may be touched only once that CTA runs.  Every thread of the cluster says so as soon as
// its CTA is set up (nothing is released: what a CTA writes for others is ordered by a later meeting) and waits for the others
// right before the first store to one of them, long after they have said it.
__device__ __forceinline__ void cluster_say_begun() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_begun() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// 32 consecutive 32-bit columns of this thread's lane (warp w of a warpgroup reads lanes 32 (w % 4) ..).
__device__ __forceinline__ void tmem_load_32x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_load_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

}  // namespace sm100
