// Exact Goldilocks linear maps on the integer tensor cores (sm_100a tcgen05,
// kind::i8): the pieces that the Tip5 MDS (tip5_mma.cuh) and the LDE's register
// transforms (lde_mma.cu) share.
//
// A linear map y = W x over the field with constant W is an integer GEMM of
// bytes: A holds 128 rows of x (64-bit words, any representatives, little
// endian), B holds B[8 r + t][8 c + b] = byte t of (W[r][c] * 2^(8 b) mod p), and
// the 32-bit accumulators D[8 r + t] give y_r = sum_t D[8 r + t] * 2^(8 t) (mod p).
// It is exact as long as a row's accumulators stay below 2^24 (mma8_recombine).
//
// Waits are bounded: after MMA8_WAIT_CYCLES a thread counts a timeout
// (g_mma8_timeouts) and its group stops issuing; the kernel then runs to its
// end, waits once more (bounded too) for the MMA it gave up on, frees its TMEM and
// returns.
#pragma once
#include <cstdint>
#include "bounded_wait.h"
#include "field.cuh"

namespace tvmc {

constexpr long long MMA8_WAIT_CYCLES = 1ll << 31;  // about one second
static __device__ unsigned int g_mma8_timeouts = 0;

// sum_t d[t] * 2^(8 t) (mod p), canonical, for d[t] < 2^24 with d[0] + 256 d[1],
// d[2] + 256 d[3], ... and d[4] + 256 d[5] + 2^16 all below 2^32.  Pairs and then
// 32-bit limbs: T = L0 + L1 * 2^32 + L2 * 2^64 with L2 < 2^17, and T = L + Z, Z =
// L2 * (2^32 - 1), is formed as L - (p - Z) with p added back on a borrow; p - Z
// has the limbs (L2 + 1, ~L2).  Without a borrow the result is L + Z - p <
// 2^32 + 2^49, with one it is L + Z < p: canonical either way.
__device__ __forceinline__ uint64_t mma8_recombine(const uint32_t* d) {
    const uint32_t p0 = d[0] + (d[1] << 8), p1 = d[2] + (d[3] << 8);
    const uint32_t p2 = d[4] + (d[5] << 8), p3 = d[6] + (d[7] << 8);
    const uint32_t a = p2 + (p1 >> 16);
    uint32_t r0, r1;
    asm("{\n\t"
        ".reg .u32 t, u, v, l0, l1, n0, n1, m;\n\t"
        "shl.b32 t, %3, 16;\n\t"
        "shl.b32 u, %5, 16;\n\t"
        "shr.u32 v, %5, 16;\n\t"
        "add.cc.u32 l0, %2, t;\n\t"
        "addc.cc.u32 l1, %4, u;\n\t"
        "addc.u32 n0, v, 1;\n\t"
        "neg.s32 n1, n0;\n\t"
        "sub.cc.u32 l0, l0, n0;\n\t"
        "subc.cc.u32 l1, l1, n1;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 %0, l0, m;\n\t"
        "subc.u32 %1, l1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1)
        : "r"(p0), "r"(p1), "r"(a), "r"(p3));
    return ((uint64_t)r1 << 32) | r0;
}

// K-major operand descriptors: rows of 128 bytes with the 128-byte swizzle
// (8-row groups 1024 bytes apart), or unswizzled 8 x 16-byte core matrices
// (128 bytes apart along K, 8-row groups 256 bytes apart).
__device__ __forceinline__ uint64_t mma8_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t mma8_desc_plain(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (8ull << 16) | (16ull << 32) | (1ull << 46);
}
// Byte offset of 64-bit word w of row r in a tile of 128-byte rows with the
// 128-byte swizzle (tile on a 1024-byte boundary).
__device__ __forceinline__ uint32_t mma8_sw128(uint32_t r, uint32_t w) {
    return 128 * r + (((w >> 1) ^ (r & 7)) << 4) + 8 * (w & 1);
}

// One K = 32 step: s32 accumulators, unsigned bytes on both sides, M = 128.
template <int N>
__device__ __forceinline__ void mma8_step(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    constexpr uint32_t idesc = (2u << 4) | (((uint32_t)N >> 3) << 17) | ((128u >> 4) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The mbarrier at `bar` completes when the MMAs issued so far by this thread do.
__device__ __forceinline__ void mma8_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Orders this thread's shared-memory writes and TMEM loads before the MMAs that
// a thread of the group issues after the barrier `id` of `threads` threads.
__device__ __forceinline__ void mma8_ready(int id, int threads) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void mma8_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ bool mma8_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Waits for the group's MMAs (whole warps together).
__device__ __forceinline__ void mma8_wait(uint32_t bar, GroupWaits& w) {
    if (!group_wait(w, [&](uint32_t parity) { return mma8_try_wait(bar, parity); }, [] { return clock64(); },
                    MMA8_WAIT_CYCLES))
        atomicAdd(&g_mma8_timeouts, 1u);
    __syncwarp();
    mma8_after();
}
// The group's issuing thread, before the barrier that precedes mma8_free.
__device__ __forceinline__ void mma8_drain(uint32_t bar, const GroupWaits& w) {
    group_drain(w, [&](uint32_t parity) { return mma8_try_wait(bar, parity); }, [] { return clock64(); },
                MMA8_WAIT_CYCLES);
}

// 32 consecutive D columns of this thread's TMEM lane, complete on return (the
// wait carries the registers, so that no use of them moves above it).
#define TVMC_W8(o) "=r"(d[o]), "=r"(d[o + 1]), "=r"(d[o + 2]), "=r"(d[o + 3]), "=r"(d[o + 4]), "=r"(d[o + 5]), \
                   "=r"(d[o + 6]), "=r"(d[o + 7])
#define TVMC_RW8(o) "+r"(d[o]), "+r"(d[o + 1]), "+r"(d[o + 2]), "+r"(d[o + 3]), "+r"(d[o + 4]), "+r"(d[o + 5]), \
                    "+r"(d[o + 6]), "+r"(d[o + 7])
__device__ __forceinline__ void mma8_ld32(uint32_t (&d)[32], uint32_t a) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : TVMC_W8(0), TVMC_W8(8), TVMC_W8(16), TVMC_W8(24)
        : "r"(a));
    asm volatile("tcgen05.wait::ld.sync.aligned;" : TVMC_RW8(0), TVMC_RW8(8), TVMC_RW8(16), TVMC_RW8(24)::"memory");
}
__device__ __forceinline__ void mma8_ld16(uint32_t (&d)[16], uint32_t a) {  // valid after mma8_ld_wait
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : TVMC_W8(0), TVMC_W8(8)
        : "r"(a));
}
__device__ __forceinline__ void mma8_ld_wait(uint32_t (&d)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : TVMC_RW8(0), TVMC_RW8(8)::"memory");
}
#undef TVMC_W8
#undef TVMC_RW8

// TMEM columns for the CTA: the first warp allocates and leaves the base address
// in shared memory at `slot`; the same warp frees them.
template <int COLS>
__device__ __forceinline__ void mma8_alloc(uint32_t slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void mma8_free(uint32_t base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS));
}
__device__ __forceinline__ void mma8_init_bar(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint64_t v) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"((uint32_t)v), "r"((uint32_t)(v >> 32)) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint64_t u, uint64_t v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"((uint32_t)u), "r"((uint32_t)(u >> 32)),
                 "r"((uint32_t)v), "r"((uint32_t)(v >> 32))
                 : "memory");
}

}  // namespace tvmc
