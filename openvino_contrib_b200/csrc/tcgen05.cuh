// Thin wrappers over the sm_100a instructions the prefill kernel is built from: mbarrier, TMA (cp.async.bulk.tensor,
// each CTA loading its own tiles), tcgen05 (TMEM allocation, MMA, commit, TMEM load/store) and the shared-memory /
// instruction descriptors of the 5th-generation tensor core.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace b2a {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier -----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2^31 clock ticks (about a second) or as soon as another thread has given up, and
// raises the CTA's abort flag.  The caller must then leave its loop and head for the common exit.
constexpr long long kWaitTicks = 1LL << 31;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitTicks) {
            *abort_flag = 1;
            return false;
        }
    }
}

// ---- TMA ----------------------------------------------------------------------------------------------------
// 4-D tiled load global -> shared, completion counted in bytes on an mbarrier.  c0 is the innermost coordinate and
// must be a multiple of 8 for 16-bit elements (16-byte rule).
__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t smem_src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
                 "r"(smem_src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
// The load with an L2 cache policy (createpolicy): evict-first for data that is touched once (Q tiles), so that it does
// not push out the K/V tiles that every query head of a group comes back for.
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void tma_load_4d_hint(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2, int c3, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
        ::"r"(smem_dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// only until the stores have READ their shared-memory source (it may be overwritten; the writes may still be in flight)
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- TMEM ---------------------------------------------------------------------------------------------------
// Executed by one whole warp.  The base address (lane 0, first column) is written to shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets lane (taddr.lane + i), columns taddr.col ..+31
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
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
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// ---- descriptors --------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor (64 bits): start address >> 4 in [0,14), leading byte offset >> 4 in [16,30),
// stride byte offset >> 4 in [32,46), version 1 in [46,48), layout type in [61,64) (2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}
// Instruction descriptor of kind::f16 (32 bits): D format f32 (1) in [4,6), A format in [7,10), B format in [10,13)
// (0 = f16, 1 = bf16), A major in bit 15, B major in bit 16 (0 = K-major, 1 = MN-major), N >> 3 in [17,23),
// M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t instr_desc_f16_ab(bool a_bf16, bool b_bf16, bool b_mn_major, int m, int n) {
    return (1u << 4) | ((a_bf16 ? 1u : 0u) << 7) | ((b_bf16 ? 1u : 0u) << 10) | ((b_mn_major ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
__host__ __device__ constexpr uint32_t instr_desc_f16(bool bf16, bool b_mn_major, int m, int n) {
    return instr_desc_f16_ab(bf16, bf16, b_mn_major, m, n);
}

// D[tmem] (+)= A . B, issued by ONE thread, A in shared memory or in tensor memory.  The 64-bit descriptors are put together inside the asm block from a
// 32-bit base (low word of the descriptor of the tile's first byte), a compile-time offset in 16-byte units and a
// compile-time high word, so that the compiler has one live register per tile instead of one per MMA.
__device__ __host__ constexpr uint32_t desc_lo_sw128(uint32_t lbo_bytes) { return ((lbo_bytes >> 4) & 0x3FFFu) << 16; }
__device__ __host__ constexpr uint32_t desc_hi_sw128(uint32_t sbo_bytes) {
    return ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
}
template <uint32_t kOffA, uint32_t kOffB, uint32_t kLoA, uint32_t kLoB, uint32_t kHiA, uint32_t kHiB, uint32_t kIdesc>
__device__ __forceinline__ void mma_ss_c(uint32_t d_tmem, uint32_t a_addr16, uint32_t b_addr16, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b32 la, lb, id;\n"
        ".reg .b64 da, db;\n"
        "setp.ne.b32 p, %3, 0;\n"
        "add.u32 la, %1, %4;\n"
        "add.u32 lb, %2, %5;\n"
        "mov.b64 da, {la, %6};\n"
        "mov.b64 db, {lb, %7};\n"
        "mov.b32 id, %8;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, id, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_addr16), "r"(b_addr16), "r"(accumulate), "n"(kOffA + kLoA), "n"(kOffB + kLoB), "n"(kHiA), "n"(kHiB), "n"(kIdesc)
        : "memory");
}
template <uint32_t kOffA, uint32_t kOffB, uint32_t kLoB, uint32_t kHiB, uint32_t kIdesc>
__device__ __forceinline__ void mma_ts_c(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_addr16, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b32 ta, lb, id;\n"
        ".reg .b64 db;\n"
        "setp.ne.b32 p, %3, 0;\n"
        "add.u32 ta, %1, %4;\n"
        "add.u32 lb, %2, %5;\n"
        "mov.b64 db, {lb, %6};\n"
        "mov.b32 id, %7;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, id, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_addr16), "r"(accumulate), "n"(kOffA), "n"(kOffB + kLoB), "n"(kHiB), "n"(kIdesc)
        : "memory");
}
// Four instructions, the operands' descriptors a constant number of 16-byte units (TMEM columns) apart.  The WHOLE warp
// executes this (and mma_commit<true>), converged; one elected lane - the same every time - issues.  Descriptors and predicates are
// warp-uniform then, which is what the instruction wants: a single lane in a branch of its own moves every one of them over
// first.  Cycles of the issuing warp for eight instructions of M = N = 128, K = 16 (the tensor core takes 512): a lane in
// a branch 436, elected one by one 303, elected four a block 174; and four of them between a wait and a commit 450 and 266.
template <uint32_t kStepA, uint32_t kStepB, uint32_t kIdesc>
__device__ __forceinline__ void mma_ss_x4(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, e, t;\n"
        ".reg .b64 a1, a2, a3, b1, b2, b3;\n"
        ".reg .b32 id;\n"
        "setp.ne.b32 p, %3, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "mov.b32 id, %4;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "add.s64 a1, %1, %5;\n"
        "add.s64 a2, %1, %6;\n"
        "add.s64 a3, %1, %7;\n"
        "add.s64 b1, %2, %8;\n"
        "add.s64 b2, %2, %9;\n"
        "add.s64 b3, %2, %10;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, id, p;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, id, t;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, id, t;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, id, t;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(accumulate), "n"(kIdesc), "n"(kStepA), "n"(2 * kStepA), "n"(3 * kStepA), "n"(kStepB),
        "n"(2 * kStepB), "n"(3 * kStepB)
        : "memory");
}
// the same with A in tensor memory
template <uint32_t kStepA, uint32_t kStepB, uint32_t kIdesc>
__device__ __forceinline__ void mma_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, e, t;\n"
        ".reg .b64 b1, b2, b3;\n"
        ".reg .b32 id, a1, a2, a3;\n"
        "setp.ne.b32 p, %3, 0;\n"
        "setp.eq.b32 t, 0, 0;\n"
        "mov.b32 id, %4;\n"
        "elect.sync _|e, 0xffffffff;\n"
        "add.u32 a1, %1, %5;\n"
        "add.u32 a2, %1, %6;\n"
        "add.u32 a3, %1, %7;\n"
        "add.s64 b1, %2, %8;\n"
        "add.s64 b2, %2, %9;\n"
        "add.s64 b3, %2, %10;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, id, p;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, id, t;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, id, t;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, id, t;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(accumulate), "n"(kIdesc), "n"(kStepA), "n"(2 * kStepA), "n"(3 * kStepA), "n"(kStepB),
        "n"(2 * kStepB), "n"(3 * kStepB)
        : "memory");
}
// the mbarrier receives one arrival when every MMA issued so far by this thread, or the warp's elected lane, has completed
template <bool kWarp>
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    if constexpr (kWarp) {
        asm volatile(
            "{\n"
            ".reg .pred e;\n"
            "elect.sync _|e, 0xffffffff;\n"
            "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
            "}\n" ::"r"(bar)
            : "memory");
    } else {
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    }
}

}  // namespace tc
}  // namespace b2a
