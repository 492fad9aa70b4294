// PTX wrappers of the tcgen05 kernels (quantized matmul and its input gradient): mbarriers with
// bounded waits, TMA tile copies, tensor-memory allocation and access, tcgen05.mma and its
// descriptors.
#pragma once
#include <cuda.h>

#include "bw_common.cuh"

namespace bw {
namespace umma {

constexpr unsigned UMMA_WAIT_LIMIT = 1u << 22;   // polls of >= 20 ns each: gives up after ~0.1-1 s

// ---- PTX wrappers ----------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Non-blocking test of a phase (the bounded loop around it does the waiting).
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false (and records the error) when the limit is hit or another
// thread of the CTA has already given up.  The thread that hits the limit stays a few milliseconds: the CTA gives
// nothing back before it has reached the closing barrier, and copies into its shared memory and MMAs into its tensor
// memory may still be in flight (microseconds).  (A look at the flag behind that barrier instead cost every launch of
// a 48-token layer 0.4 us.)
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, volatile int *abort_flag, int code, int *status) {
    unsigned tries = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (*abort_flag) return false;
        __nanosleep(20);
        if (++tries > UMMA_WAIT_LIMIT) {
            *abort_flag = code;
            atomicExch(status, code);
            for (int i = 0; i < 4; ++i) __nanosleep(1000000);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_addr(dst)), "l"(map), "r"(smem_addr(bar)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_in_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_in_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// (The umma_* calls below are made by all lanes of the issuing warp; one elected lane issues.)
// Both operands in shared memory.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Same MMA with the A operand (128 rows x 16 k, two fp16 per 32-bit column, one row per lane) in
// tensor memory: only the B operand is read from shared memory.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Each thread of the warp writes 32 consecutive 32-bit columns of its own TMEM lane.
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// Arrives on the mbarrier once all tcgen05.mma issued so far by this warp's elected lane have
// completed (called by all lanes of the issuing warp).
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile(
        "{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n"
        " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile whose rows are 128 bytes (64 fp16)
// stored with the 128-byte swizzle: 8-row groups are 1024 bytes apart (stride byte offset), the
// leading byte offset is unused for swizzled K-major layouts, descriptor version 1 (sm_100),
// layout type 2 (SWIZZLE_128B).  `addr` may be advanced by 32 bytes per 16-element k step.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);          // bits [0,14): start address >> 4
    d |= (uint64_t)1 << 16;                           // bits [16,30): leading byte offset >> 4 (ignored)
    d |= (uint64_t)(1024u >> 4) << 32;                // bits [32,46): stride byte offset >> 4
    d |= (uint64_t)1 << 46;                           // bits [46,48): descriptor version
    d |= (uint64_t)2 << 61;                           // bits [61,64): SWIZZLE_128B
    return d;
}
// The same for an MN-major operand (the non-reduced dimension is contiguous): blocks of 64 elements of that
// dimension (128 bytes, 128-byte swizzle) x all reduction steps of the stage, one 128-byte row per step.
// Eight rows make a 1024-byte swizzle atom (stride byte offset between atoms); `block_bytes` apart lies the
// next block of 64 elements (leading byte offset).  A 16-step MMA advances `addr` by 2048 bytes.
__device__ __forceinline__ uint64_t umma_smem_desc_mn(uint32_t addr, uint32_t block_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(block_bytes >> 4) << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// Instruction descriptor for kind::f16 with fp32 accumulators, M = 128, N = bn: both operands fp16 or both
// bf16 (mixed formats raise an illegal instruction); `a_mn_major`: A is stored with its rows contiguous.
__device__ __forceinline__ uint32_t umma_idesc_f16(int bn, bool bf16, bool a_mn_major) {
    uint32_t d = 0;
    d |= 1u << 4;                                     // c_format = F32
    d |= (bf16 ? 1u : 0u) << 7;                       // a_format: 0 = F16, 1 = BF16
    d |= (bf16 ? 1u : 0u) << 10;                      // b_format
    d |= (a_mn_major ? 1u : 0u) << 15;                // a_major: 0 = K, 1 = MN
    d |= (uint32_t)(bn >> 3) << 17;                   // n_dim
    d |= (uint32_t)(128 >> 4) << 24;                  // m_dim
    return d;
}

}  // namespace umma
}  // namespace bw
