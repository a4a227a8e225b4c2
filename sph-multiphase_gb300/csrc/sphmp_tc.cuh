// sphmp_tc.cuh — fifth-generation tensor-core primitives for sm_103a, in inline
// PTX: tensor-memory (TMEM) allocation, shared-memory matrix descriptors,
// tcgen05.mma of kind::f16 (bf16 operands, FP32 accumulators in TMEM), the
// commit to an mbarrier and a bounded wait on it, and tcgen05.ld of the
// accumulators.
//
// Operand layout: K-major without swizzling. A tile of R rows (M or N) and Kc
// columns (bf16) is stored as 8 x 8 core matrices of 128 contiguous bytes
// (8 rows of 16 bytes); core matrices adjacent in K are 128 bytes apart (the
// leading-dimension byte offset), groups of 8 rows are Kc * 16 bytes apart (the
// stride-dimension byte offset). Element (r, k) lives at kmajor_offset(r, k, Kc).
// One MMA consumes K = 16 (two core matrices along K); the next one starts
// 256 bytes further.
//
// Accumulator layout for M = 128 with one CTA: row m of D is TMEM lane m,
// column n is TMEM column (base + n). Warp w of the CTA reads lanes
// [32 (w % 4), 32 (w % 4) + 32).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sphmp {
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t kmajor_offset(int r, int k, int kc) {
    return (uint32_t)((r >> 3) * (kc * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// Shared-memory matrix descriptor: start address, leading- and stride-dimension
// byte offsets (all in 16-byte units, 14 bits each), descriptor version 1
// (bits 46-47), base offset 0, no swizzling (bits 61-63 = 0).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ uint64_t kmajor_desc(uint32_t tile_addr, int kc, int kstep) {
    return smem_desc(tile_addr + (uint32_t)kstep * 256u, 128u, (uint32_t)kc * 16u);
}

// The same core matrices read the other way: an operand whose M (or N) index runs
// along the 16 contiguous bytes and whose K index runs down the 8 rows (MN-major).
// A tile [r][c] of kc columns stored for K-major use thus also serves as the operand
// of its transpose: the stride between core matrices along M / N (128 bytes) goes
// into the stride-dimension offset, the one along K (a group of 8 rows) into the
// leading-dimension offset. One MMA consumes two core matrices along K.
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t tile_addr, int kc, int kstep) {
    return smem_desc(tile_addr + (uint32_t)kstep * (uint32_t)kc * 32u, (uint32_t)kc * 16u, 128u);
}

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B bf16
// (bits 7-9 = 1, 10-12 = 1), K-major or MN-major (bits 15, 16 = 0 or 1), N / 8 in bits
// 17-22, M / 16 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int m, int n, bool a_mn = false, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- TMEM (one full warp executes alloc / dealloc) ----
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// generic-proxy shared-memory writes become visible to the tensor core
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- MMA, issued by one thread ----
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// the mbarrier receives one arrival when every MMA issued before has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_addr(bar))
                 : "memory");
}

// ---- mbarrier ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait until the phase of parity `parity` has completed, for at most
// `limit_ns` nanoseconds; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
    const uint32_t a = smem_addr(bar);
    const uint64_t t0 = global_ns();
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// ---- accumulator loads: 16 consecutive columns of this thread's lane ----
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive columns of this thread's lane, queued: r holds them after
// tmem_wait16 (which takes r, so that no use of it moves before the wait).
__device__ __forceinline__ void tmem_issue16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
        :
        : "memory");
}

// TMEM address of column `col` in the lane quadrant of warp `warp`
__device__ __forceinline__ uint32_t tmem_lane_addr(uint32_t base, int warp, int col) {
    return base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col;
}

constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s: an MMA of these sizes takes microseconds

}  // namespace tc
}  // namespace sphmp
