// Tip5 permutation with the MDS layer on the tensor cores (sm_100a tcgen05).
//
// The MDS is the one dense contraction of the path: 16 words x a constant
// 16 x 16 matrix, per state.  Both sides are split into bytes, so that it is an
// exact integer GEMM of kind::i8 (unsigned bytes, 32-bit accumulators):
//
//   A  128 states x 128 bytes   (a state's 16 words, little endian, one row per
//                                state)
//   B  128 x 128 bytes          B[8 r + t][8 c + b] = byte t of
//                                (M[(r - c) mod 16] * 2^(8 b) mod p)
//   D  128 x 128 (TMEM, s32)    D[8 r + t] = sum over c, b
//
// so output word r is sum_t D[8 r + t] * 2^(8 t) (mod p).  Taking the weights
// mod p keeps them in eight bytes (only b = 7 needs it: M = 256 M1 + M0 gives
// M0 * 2^56 + M1 * (2^32 - 1)), so N = 128 and four groups of 128 states fill the
// SM's 512 TMEM columns exactly.  At most three nonzero digits per (c, t) bound
// every D below 16 * 3 * 255^2 + 255 < 2^22.  The round constants come from one
// more K = 32 step, ones(128 x 32) x their bytes, so they cost no instruction of
// the threads.
//
// What bounds it: the integer pipes, in x^7 (69 instructions a word) and in the
// recombination (17 a word): multiply-add 71% and ALU 64% busy, an instruction
// issued in 63% of the cycles.  Against an MDS on the FP64 pipe
// this takes 336 FP64 instructions and the recombination of two 52-bit halves
// out of a round; what it adds is a shared-memory store of the state, one barrier
// of the group and the MMA's latency, which the SM's other three groups cover
// (tensor pipe 16% busy).  Two threads share a state: 64 registers each, 32 warps
// per SM.  227328 rows x 379 (three full waves of tiles), B200: the FP64 kernel
// (one thread per state, six 128-thread CTAs per SM) 2.85 ms; this one 2.40 ms.
// One thread per state with four or six groups: 2.47 and 2.49; four threads per
// state with two groups: 2.78 (too little to cover the MMA's latency).
#pragma once
#include <cstdint>
#include "field.cuh"
#include "mma_i8.cuh"
#include "tip5.cuh"

namespace tvmc {

constexpr int T5M_STATES = 128;                        // states per MMA (rows of A)
constexpr int T5M_PARTS = 2;                           // threads per state
constexpr int T5M_GROUP = T5M_PARTS * T5M_STATES;      // threads per group
constexpr int T5M_GROUPS = 4;                          // groups per CTA
constexpr int T5M_THREADS = T5M_GROUP * T5M_GROUPS;
constexpr int T5M_COLS = 128 * T5M_GROUPS;             // TMEM columns
constexpr int T5M_WORDS = T5_STATE / T5M_PARTS;        // words per thread
constexpr int T5M_LOOKUPS = 4 / T5M_PARTS;             // of which lookups

// Part q of a state holds lookup words 2 q, 2 q + 1 and x^7 words 4 + 6 q .. 9 + 6 q:
// the same work for both.  The state word of its i-th; in A, B and D word
// t5m_word(q, i) has position 8 q + i, so that a part's bytes and accumulators
// are contiguous.
__device__ __forceinline__ int t5m_word(int q, int i) {
    return i < T5M_LOOKUPS ? T5M_LOOKUPS * q + i : 4 + (T5M_WORDS - T5M_LOOKUPS) * q + i - T5M_LOOKUPS;
}

// Shared-memory map, as addresses in the CTA's shared window.  The byte table
// sits on a 64 KB boundary, entry v of lane l at v * 256 + l * 4, so that one
// byte permute of (word, lane base) is the whole address of a lookup.
constexpr uint32_t T5M_SBOX = 0x10000;                 // 64 KB
constexpr uint32_t T5M_A = 0x20000;                    // 4 x 16 KB, rows of 128 bytes, 128-byte swizzle
constexpr uint32_t T5M_END = T5M_A + T5M_GROUPS * 0x4000;
// below the table, from the (1024-byte aligned) start of the dynamic region:
constexpr uint32_t T5M_B = 0;                          // 16 KB, 128-byte swizzle
constexpr uint32_t T5M_ONES = 0x4000;                  // 4 KB, no swizzle
constexpr uint32_t T5M_RC = 0x5000;                    // 5 x 4 KB, no swizzle
constexpr uint32_t T5M_BAR = 0xA000;                   // one mbarrier per group
constexpr uint32_t T5M_TMEM = T5M_BAR + 32;            // TMEM base address
constexpr uint32_t T5M_BYTES = T5M_END;                // dynamic shared memory: the map from address 0

// The constant operand images: B (word w of row n at [16 n + w], by position) and
// byte t of word r's round constants, in Montgomery form, at [round][8 r + t].
struct T5mImages {
    uint64_t b[T5M_STATES * T5_STATE];
    uint32_t rc[T5_ROUNDS * T5M_STATES];
};
constexpr int t5m_at_const(int pos) {
    const int q = pos / T5M_WORDS, i = pos % T5M_WORDS;
    return i < T5M_LOOKUPS ? T5M_LOOKUPS * q + i : 4 + (T5M_WORDS - T5M_LOOKUPS) * q + i - T5M_LOOKUPS;
}
constexpr T5mImages t5m_images() {
    const uint64_t col[T5_STATE] = {TVMC_T5_MDS_FIRST_COLUMN};
    const T5RcMont rc = t5_rc_mont();
    T5mImages im{};
    for (int n = 0; n < T5M_STATES; n++) {
        const int r = t5m_at_const(n >> 3), t = n & 7;
        for (int w = 0; w < T5_STATE; w++) {
            const uint64_t m = col[(r - t5m_at_const(w)) & 15];
            uint64_t v = 0;
            for (int b = 0; b < 8; b++) {
                const uint64_t x = b < 7 ? m << (8 * b) : (m << 56) + (m >> 8) * 0xFFFFFFFFull;
                v |= ((x >> (8 * t)) & 0xFF) << (8 * b);
            }
            im.b[16 * n + w] = v;
        }
        for (int rnd = 0; rnd < T5_ROUNDS; rnd++)
            im.rc[T5M_STATES * rnd + n] = (uint32_t)(rc.v[rnd * T5_STATE + r] >> (8 * t)) & 0xFF;
    }
    return im;
}
static __device__ const T5mImages g_t5m_images = t5m_images();

// What a thread keeps of its group's MMA.
struct T5Mma {
    uint32_t base;     // start of the low part of the shared map
    uint32_t a[T5M_WORDS / 2];  // shared addresses of this thread's word pairs in its A row
    uint32_t sbox;     // T5M_SBOX + lane * 4
    uint32_t tmem;     // this warp's lanes of the group's D columns
    GroupWaits waits;
    int group;
    int row;           // this thread's state within the group
    int part;          // and its part of it
};

// Value of the S-box table for a 32-bit word, byte by byte: the permute puts
// byte k of m between the lane's offset and the table's address.
__device__ __forceinline__ uint32_t t5m_lds(uint32_t a) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t t5m_lookup32(uint32_t m, uint32_t sbox) {
    const uint32_t w0 = t5m_lds(__byte_perm(m, sbox, 0x7604));
    const uint32_t w1 = t5m_lds(__byte_perm(m, sbox, 0x7614));
    const uint32_t w2 = t5m_lds(__byte_perm(m, sbox, 0x7624));
    const uint32_t w3 = t5m_lds(__byte_perm(m, sbox, 0x7634));
    return __byte_perm(__byte_perm(w0, w1, 0x0040), __byte_perm(w2, w3, 0x0040), 0x5410);
}
// split_and_lookup of a canonical Montgomery-form word.
__device__ __forceinline__ uint64_t t5m_split_lookup(uint64_t x, uint32_t sbox) {
    const uint32_t y0 = t5m_lookup32((uint32_t)x, sbox), y1 = t5m_lookup32((uint32_t)(x >> 32), sbox);
    return ((uint64_t)y1 << 32) | y0;
}

// The 128-bit product with the diagonal products formed whole (mul.wide: four
// cycles of the multiply-add pipe against six for a low and a high product) and
// the cross products added onto the middle limbs.  x^7 of a warp, alone on a
// full SM: 123 -> 116 cycles against gl_mul128 (in the LDE kernels, whose
// registers are scarcer, it measured 4% slower).
__device__ __forceinline__ void t5m_mul128(uint64_t a, uint64_t b, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                           uint32_t& r3) {
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    asm("{\n\t"
        ".reg .u64 p, q;\n\t"
        ".reg .u32 p1, q0, q1;\n\t"
        "mul.wide.u32 p, %4, %6;\n\t"
        "mul.wide.u32 q, %5, %7;\n\t"
        "mov.b64 {%0, p1}, p;\n\t"
        "mov.b64 {q0, q1}, q;\n\t"
        "mad.lo.cc.u32 p1, %4, %7, p1;\n\t"
        "madc.hi.cc.u32 q0, %4, %7, q0;\n\t"
        "addc.u32 q1, q1, 0;\n\t"
        "mad.lo.cc.u32 %1, %5, %6, p1;\n\t"
        "madc.hi.cc.u32 %2, %5, %6, q0;\n\t"
        "addc.u32 %3, q1, 0;\n\t"
        "}"
        : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
        : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
}

// x^7 of a Montgomery-form word (t5_pow7_m); any 64-bit representative in and out.
__device__ __forceinline__ uint64_t t5m_pow7(uint64_t x) {
    uint32_t r0, r1, r2, r3;
    gl_sqr128(x, r0, r1, r2, r3);
    const uint64_t x2 = gl_redc(r0, r1, r2, r3);
    t5m_mul128(x, x2, r0, r1, r2, r3);
    const uint64_t x3 = gl_redc(r0, r1, r2, r3);
    gl_sqr128(x2, r0, r1, r2, r3);
    const uint64_t x4 = gl_redc(r0, r1, r2, r3);
    t5m_mul128(x3, x4, r0, r1, r2, r3);
    return gl_redc(r0, r1, r2, r3);
}

// Every thread of the CTA calls this once, before anything else: tables,
// operand tiles, barriers and the TMEM columns.
__device__ __forceinline__ void t5m_init(T5Mma& c, uint32_t dyn) {
    c.base = (dyn + 1023) & ~1023u;
    const int tid = threadIdx.x;
    if (tid < 32) mma8_alloc<T5M_COLS>(c.base + T5M_TMEM);
    if (tid < T5M_GROUPS) mma8_init_bar(c.base + T5M_BAR + 8 * tid);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int i = tid; i < T5_SBOX_WORDS; i += T5M_THREADS)
        sts32(T5M_SBOX + (i >> 5) * 256 + (i & 31) * 4, __ldg(&g_t5_sbox.v[i >> 5]));
    // ones and round-constant tiles: byte k = 0 of every row, zero elsewhere
    for (int i = tid; i < 6 * 256; i += T5M_THREADS) {  // 16-byte chunk j of row n of a tile
        const int tile = i >> 8, n = (i >> 1) & 127, j = i & 1;
        const uint32_t v = j ? 0u : (tile == 0 ? 1u : __ldg(&g_t5m_images.rc[T5M_STATES * (tile - 1) + n]));
        sts128(c.base + T5M_ONES + tile * 4096 + (n >> 3) * 256 + j * 128 + (n & 7) * 16, v, 0);
    }
    for (int i = tid; i < T5M_STATES * T5_STATE; i += T5M_THREADS)
        sts64(c.base + T5M_B + mma8_sw128(i >> 4, i & 15), __ldg(&g_t5m_images.b[i]));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tb = lds32(c.base + T5M_TMEM);
    c.row = tid & (T5M_STATES - 1);
    c.group = tid / T5M_GROUP;
    c.part = (tid / T5M_STATES) % T5M_PARTS;
#pragma unroll
    for (int i = 0; i < T5M_WORDS; i += 2)
        c.a[i / 2] = T5M_A + 16384 * c.group + mma8_sw128(c.row, T5M_WORDS * c.part + i);
    c.sbox = T5M_SBOX + (tid & 31) * 4;
    asm volatile("" : "+r"(c.sbox)::"memory");  // no lookup moves above the barrier
    c.tmem = tb + 128 * c.group + 8 * T5M_WORDS * c.part + ((uint32_t)(c.row & ~31) << 16);
    c.waits = GroupWaits{};
}

// Every thread of the CTA calls this last.
__device__ __forceinline__ void t5m_done(const T5Mma& c) {
    if ((threadIdx.x & (T5M_GROUP - 1)) == 0) mma8_drain(c.base + T5M_BAR + 8 * c.group, c.waits);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        mma8_after();
        mma8_free<T5M_COLS>(lds32(c.base + T5M_TMEM));
    }
}

// MDS of the group's 128 states plus the round constants of round rnd.  All
// threads of the group call it together, each with its part of its state.
__device__ __forceinline__ void t5m_mds(uint64_t (&s)[T5M_WORDS], int rnd, T5Mma& c) {
#pragma unroll
    for (int i = 0; i < T5M_WORDS; i += 2) sts128(c.a[i / 2], s[i], s[i + 1]);
    mma8_ready(c.group + 1, T5M_GROUP);
    const uint32_t bar = c.base + T5M_BAR + 8 * c.group;
    if ((threadIdx.x & (T5M_GROUP - 1)) == 0 && !c.waits.dead) {
        mma8_after();
        const uint32_t d = c.tmem;
        mma8_step<128>(d, mma8_desc_plain(c.base + T5M_ONES), mma8_desc_plain(c.base + T5M_RC + 4096 * rnd), 0);
        const uint64_t da = mma8_desc_sw128(T5M_A + 16384 * c.group), db = mma8_desc_sw128(c.base + T5M_B);
#pragma unroll
        for (int k = 0; k < 4; k++) mma8_step<128>(d, da + 2 * k, db + 2 * k, 1);
        mma8_commit(bar);
    }
    mma8_wait(bar, c.waits);
#pragma unroll
    for (int h = 0; h < T5M_WORDS; h += 4) {
        uint32_t d[32];
        mma8_ld32(d, c.tmem + 8 * h);
#pragma unroll
        for (int i = 0; i < 4; i++) s[h + i] = mma8_recombine(d + 8 * i);
    }
}

// The permutation of the group's 128 states, canonical Montgomery form in
// (words 0-3; any representative in words 4-15) and canonical out.
__device__ __forceinline__ void t5m_permutation(uint64_t (&s)[T5M_WORDS], T5Mma& c) {
#pragma unroll 1
    for (int rnd = 0; rnd < T5_ROUNDS; rnd++) {
#pragma unroll
        for (int i = 0; i < T5M_LOOKUPS; i++) s[i] = t5m_split_lookup(s[i], c.sbox);
#pragma unroll
        for (int i = T5M_LOOKUPS; i < T5M_WORDS; i++) s[i] = t5m_pow7(s[i]);
        t5m_mds(s, rnd, c);
    }
}

}  // namespace tvmc
