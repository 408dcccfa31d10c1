// PTX wrappers of the tcgen05 kernels: mbarriers with bounded waits, TMA, tensor memory, descriptors.
#pragma once
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "ring.cuh"

namespace mtc {

constexpr uint32_t kSpinLimit = 1u << 22;   // bounded waits: ~seconds, then give up

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// try_wait with a suspend-time hint: the thread may sleep in hardware for up to `ns` before it reports failure
__device__ __forceinline__ bool mbar_try_hint(uint64_t *bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(ns) : "memory");
    return ok != 0;
}
// Polls until the phase completes: 1; the abort flag is set: 2; neither within kSpinLimit polls: 0.  Sixteen polls of two instructions
// each between two looks at the flag: with a loop around a single poll the waiting warps issued more instructions than the working ones.
__device__ __forceinline__ uint32_t mbar_poll(uint32_t bar, uint32_t parity, uint32_t abort) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 i, f;\n\t"
        "mov.u32 %0, 1;\n\t"
        "mov.u32 i, %4;\n\t"
        "POLL:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE;\n\t"
        "ld.volatile.shared.u32 f, [%3];\n\t"
        "mov.u32 %0, 2;\n\t"
        "setp.ne.u32 p, f, 0;\n\t@p bra DONE;\n\t"
        "mov.u32 %0, 1;\n\t"
        "sub.u32 i, i, 1;\n\t"
        "setp.ne.u32 p, i, 0;\n\t@p bra POLL;\n\t"
        "mov.u32 %0, 0;\n\t"
        "DONE:\n\t}"
        : "=&r"(r) : "r"(bar), "r"(parity), "r"(abort), "n"(kSpinLimit / 16) : "memory");
    return r;
}
// Bounded wait.  Returns false when the barrier did not complete within kSpinLimit polls (the CTA's abort flag and the global status
// word are raised then) or another role already aborted.  `sleep_ns` > 0 lets the hardware suspend the thread between polls.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort, uint32_t *status, uint32_t code,
                                          uint32_t sleep_ns = 0) {
    if (sleep_ns) {
        for (uint32_t i = 0; i < kSpinLimit; ++i) {
            if (mbar_try_hint(bar, parity, sleep_ns)) return true;
            if ((i & 63u) == 63u && *abort) return false;
        }
    } else {
        const uint32_t r = mbar_poll(smem_u32(bar), parity, smem_u32(const_cast<uint32_t *>(abort)));
        if (r) return r == 1;
    }
    *abort = 1;
    atomicCAS(status, 0u, code);
    return false;
}
// Whole-warp wait.  All lanes poll together, one instruction for the warp: with lane 0 polling and broadcasting, the other
// lanes' yields and the reconvergence after every poll were on the path of every hand-off.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile uint32_t *abort, uint32_t *status, uint32_t code,
                                               uint32_t sleep_ns = 0) {
    const bool ok = mbar_wait(bar, parity, abort, status, code, sleep_ns);
    __syncwarp();
    return ok;
}
// The same for a loop whose counters and addresses have to stay warp-uniform (the issue of MMAs): the outcome is a vote.
__device__ __forceinline__ bool mbar_wait_vote(uint64_t *bar, uint32_t parity, volatile uint32_t *abort, uint32_t *status, uint32_t code) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort, status, code));
}

// On the way out of a launch that gave up, by one thread once every role has ended: bounded waits for the copies (or MMAs) that are still on their way.
static __device__ __noinline__ void drain_ring(uint64_t *bars, uint32_t issued, int slots) {
    for (int b = 0; b < slots; ++b) {
        const int parity = ring::last_parity(issued, slots, b);
        for (uint32_t i = 0; parity >= 0 && i < 1u << 16 && !mbar_try(&bars[b], parity); ++i) {}
    }
}

// Waits and arrivals of loops that keep the barriers' shared-memory addresses: `abort` is the address of the CTA's abort flag.
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
static __device__ __noinline__ void mbar_gave_up(uint32_t outcome, uint32_t abort, uint32_t *status, uint32_t code) {
    if (outcome == 2) return;                // another role did
    asm volatile("st.volatile.shared.u32 [%0], 1;" ::"r"(abort) : "memory");
    atomicCAS(status, 0u, code);
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t abort, uint32_t *status, uint32_t code) {
    const uint32_t r = mbar_poll(bar, parity, abort);
    if (__builtin_expect(r != 1, 0)) {
        mbar_gave_up(r, abort, status, code);
        return false;
    }
    return true;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar)) : "memory");
}

// `bytes` from global to shared memory, both 16-byte aligned, a multiple of 16
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row atoms 1024 B apart.
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);   // start address  [0,14)
    d |= static_cast<uint64_t>(1) << 16;                   // leading byte offset (unused with 128B swizzle)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;           // stride byte offset [32,46)
    d |= static_cast<uint64_t>(1) << 46;                   // descriptor version (sm_100)
    d |= static_cast<uint64_t>(2) << 61;                   // SWIZZLE_128B
    return d;
}

// A from tensor memory, B from shared memory
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// tcgen05.ld / .st of the calling warp's 32 lanes x COLS columns: thread = lane, register = column
template <int COLS>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t *v) {
    static_assert(COLS == 16 || COLS == 32, "columns of one load");
    if constexpr (COLS == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
              "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr) : "memory");
}
// all 512 columns of an SM's tensor memory, for a kernel that runs one CTA an SM; one warp calls each
__device__ __forceinline__ void tmem_alloc_all(uint32_t *base) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(base)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free_all(uint32_t base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512));
}

// A row-major [rows, cols] tensor with boxes of box_rows x box_cols (128, 64 or 32 bytes) and the swizzle of that width; what lies past the ends reads as zero
cudaError_t make_map_2d(CUtensorMap *map, CUtensorMapDataType type, int elem_bytes, const void *base, long long rows, long long cols,
                        int box_rows, int box_cols, std::string *why);
// The same tensor of 16-bit elements as [cols / 64][rows][64]: one box of box_blocks x box_rows x 64 is box_blocks tiles behind each other
cudaError_t make_map_blocks(CUtensorMap *map, const void *base, long long rows, long long cols, int box_rows, int box_blocks, std::string *why);

}  // namespace mtc
