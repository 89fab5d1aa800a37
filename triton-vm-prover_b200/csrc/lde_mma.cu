// LDE and NTT passes with 2^8- or 2^10-point sub-transforms on the integer
// tensor cores.
//
// A sub-transform of N = R * R points, R = 16 or 32, is two rounds of radix R
// (ntt.cu, sub_dft).  A radix-R DFT over the field is a constant R x R map, so
// here it is an exact byte GEMM (mma_i8.cuh): 128 lines of R words form A
// (128 x 8 R bytes), the DFT matrix B is 8 R x 8 R bytes (16 or 64 KB, copied in
// once per CTA), and D is 128 x 8 R in TMEM.  A radix-32 register network costs
// about 55 instructions per element (80 butterflies of an addition and a
// shift-twiddled subtraction over 32 elements); the MMA form leaves the
// recombination of eight 32-bit accumulators, 17, and takes inputs of any
// representative, so that nothing is canonicalised on the way in.  The tensor
// pipe needs 1024 cycles per 4096 elements and round at R = 32 (256 per 2048 at
// R = 16), about a third of what the twiddle products and the recombination take.
//
// A group of 512 (R = 32) or 256 threads owns a tile of 128 lines (4 or 8
// sequences), its A tile and 8 R TMEM columns; the two or four groups of a CTA
// (one CTA per SM) work on different columns or tiles, so that the others compute
// while one waits for its MMA.  TMEM lane = line; R / 8 threads share a line, part
// q holding outputs 8 q .. 8 q + 7.  The A tile is also the transpose buffer
// between the two rounds: lines are ordered t + SEQS * d (t: sequence, d: digit),
// so that the final global accesses come in runs of SEQS words (one or two
// 32-byte sectors), except where a sequence is contiguous in memory (d + R * t).
//
// B200: LDE x4 of 32 x 2^20 3.04 -> 1.97 ms, 256 x 2^18 7.15 -> 3.57, 256 x 2^16 1.31 -> 0.85.
// D is read 16 columns at a time (32 at a time: 2.03 against 1.95 ms), the next 16
// while the current ones are recombined (128 x 2^16 0.453 -> 0.431 ms).  What bounds
// it: the twiddle products and recombinations on the integer pipes (60% and 40%
// busy) and the MMA's latency, which the other groups cover only in part.
#include "lde_mma.h"
#include "mma_i8.cuh"

namespace tvmc {

constexpr int LM_LINES = 128;              // lines per tile: TMEM lanes
constexpr int LM_THREADS = 1024;           // per CTA

// Sizes and shared memory (from the 1024-byte aligned start of the dynamic
// region) of the passes with sub-transforms of 2^(2 B) = R * R points.
template <int B>
struct LmCfg {
    static constexpr int R = 1 << B, N = R * R;
    static constexpr int SEQS = LM_LINES / R;             // sequences per tile
    static constexpr int PARTS = R / 8;                   // threads per line, eight outputs each
    static constexpr int GROUP = LM_LINES * PARTS, GROUPS = LM_THREADS / GROUP;
    static constexpr int COLS = 8 * R;                    // TMEM columns per group
    static_assert(COLS * GROUPS == 512, "all of TMEM");
    static constexpr int TWP = R + 1;                     // padded row of an R x R twiddle table
    static constexpr uint32_t A_HALF = 128 * LM_LINES, B_HALF = 128 * COLS;  // 128 bytes of K
    static constexpr uint32_t A_BYTES = A_HALF * (R / 16), B_BYTES = B_HALF * (R / 16);
    static constexpr uint32_t O_B = 0;
    static constexpr uint32_t O_A = O_B + B_BYTES;        // one tile per group
    static constexpr uint32_t O_TW = O_A + GROUPS * A_BYTES;         // w_N^(d k) at [d * TWP + k]
    static constexpr uint32_t O_TWQ = O_TW + (8 * R * TWP + 255) / 256 * 256;  // inter-pass twiddles, SEQS * N words
    static constexpr uint32_t O_BAR = O_TWQ + 8 * SEQS * N;          // mbarriers, TMEM base
    static constexpr uint32_t BYTES = O_BAR + 64;
    static constexpr uint32_t O_SCL = BYTES;              // k_lde_mid_mma: per coset [t * TWP + k1]
    static constexpr uint32_t SCL_BYTES = 8 * SEQS * TWP;
    static constexpr uint32_t TWC_BYTES = 8 * R * TWP;    // and per coset [d * TWP + k]
    static constexpr uint32_t mid_bytes(int le) { return BYTES + (1u << le) * (SCL_BYTES + TWC_BYTES); }
};
constexpr uint32_t LM_SLACK = 1024;                       // for the alignment of the base
constexpr bool lm_mid_fits(uint32_t bytes) { return bytes + LM_SLACK <= 227 * 1024; }
static_assert(lm_mid_fits(LmCfg<5>::mid_bytes(lde_mma_max_le(10))) && lm_mid_fits(LmCfg<4>::mid_bytes(lde_mma_max_le(8))),
              "the per-coset tables fit one SM");

namespace {

extern __shared__ uint8_t lm_smem[];

struct Lm {
    uint8_t* sm;     // shared map
    uint8_t* a;      // the group's A tile
    uint32_t base;   // shared address of the map
    uint32_t tmem;   // this thread's D columns in its warp's lanes
    uint32_t bar;
    GroupWaits waits;
    int group, row, part;
};

// Byte offset of word j of line r in an A tile.
template <int B>
__device__ __forceinline__ uint32_t a_word(uint32_t r, uint32_t j) {
    return (j >> 4) * LmCfg<B>::A_HALF + mma8_sw128(r, j & 15);
}
__device__ __forceinline__ uint64_t& at64(uint8_t* p) { return *reinterpret_cast<uint64_t*>(p); }

// 2^e mod p, 0 <= e < 192 (2^64 = 2^32 - 1, 2^96 = -1).
constexpr uint64_t pow2_mod(int e) {
    const int s = e >= 96 ? e - 96 : e;
    const uint64_t v = s < 64 ? 1ull << s : (1ull << (s - 32)) - (1ull << (s - 64));
    return e >= 96 ? GL_P - v : v;
}

// The DFT operand: word j of row n = 8 k + t, at [R n + j], holds byte t of
// w_R^(j k) * 2^(8 b) in its byte b (w_32 = 2^78).
template <int B>
struct DftImage {
    uint64_t w[LmCfg<B>::COLS * LmCfg<B>::R];
};
template <int B>
constexpr DftImage<B> dft_image() {
    constexpr int R = LmCfg<B>::R;
    DftImage<B> im{};
    for (int k = 0; k < R; k++)
        for (int j = 0; j < R; j++)
            for (int b = 0; b < 8; b++) {
                const uint64_t v = pow2_mod((78 * (32 / R) * j * k + 8 * b) % 192);
                for (int t = 0; t < 8; t++) im.w[R * (8 * k + t) + j] |= ((v >> (8 * t)) & 0xFF) << (8 * b);
            }
    return im;
}
static __device__ const DftImage<4> g_dft16 = dft_image<4>();
static __device__ const DftImage<5> g_dft32 = dft_image<5>();

// Every thread of the CTA calls this first.
template <int B>
__device__ __forceinline__ void lm_init(Lm& c, const uint64_t* tw12) {
    using C = LmCfg<B>;
    const uint32_t dyn = (uint32_t)__cvta_generic_to_shared(lm_smem);
    const int tid = threadIdx.x;
    c.base = (dyn + 1023) & ~1023u;
    c.sm = lm_smem + (c.base - dyn);
    if (tid < 32) mma8_alloc<512>(c.base + C::O_BAR + 32);
    if (tid < C::GROUPS) mma8_init_bar(c.base + C::O_BAR + 8 * tid);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint64_t* img;
    if constexpr (B == 4) img = g_dft16.w;
    else img = g_dft32.w;
    for (int i = tid; i < C::COLS * C::R; i += LM_THREADS) {
        const int n = i / C::R, j = i % C::R;
        at64(c.sm + C::O_B + (j >> 4) * C::B_HALF + mma8_sw128(n, j & 15)) = __ldg(img + i);
    }
    for (int i = tid; i < C::N; i += LM_THREADS) {
        const int d = i / C::R, k = i % C::R;
        at64(c.sm + C::O_TW + 8 * (d * C::TWP + k)) = gl_to_mont(__ldg(tw12 + (4096 / C::N) * d * k));
    }
    mma8_ready(0, LM_THREADS);
    mma8_after();
    c.group = tid / C::GROUP;
    c.row = tid & (LM_LINES - 1);
    c.part = (tid / LM_LINES) % C::PARTS;
    c.a = c.sm + C::O_A + C::A_BYTES * c.group;
    c.bar = c.base + C::O_BAR + 8 * c.group;
    c.tmem = lds32(c.base + C::O_BAR + 32) + C::COLS * c.group + 64 * c.part + ((uint32_t)(c.row & ~31) << 16);
    c.waits = GroupWaits{};
}

// Every thread of the CTA calls this last; sets *status if a wait ran out.
template <int B>
__device__ __forceinline__ void lm_done(const Lm& c, uint64_t* status) {
    if (c.waits.dead && status) *status = 1;
    if ((threadIdx.x & (LmCfg<B>::GROUP - 1)) == 0) mma8_drain(c.bar, c.waits);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32) {
        mma8_after();
        mma8_free<512>(lds32(c.base + LmCfg<B>::O_BAR + 32));
    }
}

// The R-point DFT of every line of the group's A tile; out(i, x) receives
// output 8 * part + i of this thread's line, canonical.  The A tile may be
// overwritten from the first out call on.
template <int B, class F>
__device__ __forceinline__ void lm_dft(Lm& c, F&& out) {
    using C = LmCfg<B>;
    mma8_ready(c.group + 1, C::GROUP);
    if ((threadIdx.x & (C::GROUP - 1)) == 0 && !c.waits.dead) {
        mma8_after();
        const uint64_t da = mma8_desc_sw128(c.base + C::O_A + C::A_BYTES * c.group), db = mma8_desc_sw128(c.base + C::O_B);
#pragma unroll
        for (int k = 0; k < C::R / 4; k++)  // 32 bytes of K, four steps per half
            mma8_step<C::COLS>(c.tmem, da + (k >> 2) * (C::A_HALF >> 4) + 2 * (k & 3),
                               db + (k >> 2) * (C::B_HALF >> 4) + 2 * (k & 3), k > 0);
        mma8_commit(c.bar);
    }
    mma8_wait(c.bar, c.waits);
    uint32_t d[2][16];
    mma8_ld16(d[0], c.tmem);
#pragma unroll
    for (int h = 0; h < 4; h++) {
        mma8_ld_wait(d[h & 1]);
        if (h < 3) mma8_ld16(d[(h + 1) & 1], c.tmem + 16 * (h + 1));
#pragma unroll
        for (int i = 0; i < 2; i++) out(2 * h + i, mma8_recombine(d[h & 1] + 8 * i));
    }
}

// This thread's eight words of its own line: four 16-byte chunks of an aligned
// group, whose swizzled addresses differ in two bits.
template <int B>
__device__ __forceinline__ void lm_fill(const Lm& c, const uint64_t (&v)[8]) {
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(c.a) + a_word<B>(c.row, 8 * c.part);
#pragma unroll
    for (int i = 0; i < 8; i += 2) sts128(a0 ^ (8 * i), v[i], v[i + 1]);
}

// Eight words of a sequence of LmCfg<B>::N at src, element k at src[k << s]: k0 + R * i,
// or with NEG the negated -(k0 + R * i) mod N.
template <int B, bool NEG>
__device__ __forceinline__ void lm_load(uint64_t (&v)[8], const uint64_t* __restrict__ src, uint32_t k0, int s) {
    using C = LmCfg<B>;
    const int64_t step = (int64_t)(NEG ? -C::R : C::R) * (1ll << s);
    const uint64_t* p = src + ((uint64_t)(NEG ? C::N - k0 : k0) << s);
    v[0] = NEG && k0 == 0 ? src[0] : *p;
#pragma unroll
    for (int i = 1; i < 8; i++) {
        p += step;
        v[i] = *p;
    }
}

// A store function of lm_dft: output i to p[R * i << s].
template <int B, class F>
__device__ __forceinline__ void lm_store(Lm& c, uint64_t* p, int s, F&& map) {
    const uint64_t step = (uint64_t)LmCfg<B>::R << s;
    lm_dft<B>(c, [&](int i, uint64_t x) {
        *p = map(i, x);
        p += step;
    });
}

__device__ __forceinline__ uint64_t tw2g(const uint64_t* __restrict__ lo, const uint64_t* __restrict__ hi, uint32_t e) {
    return gl_mul(__ldg(lo + (e & 4095)), __ldg(hi + (e >> 12)));
}

// w^((s0 + s) * k) of the tile's sequences s and points k at [SEQS * k + s]; for
// k = R * k1 + d that is [128 * k1 + row] with the lines s + SEQS * d.
template <int B>
__device__ __forceinline__ void fill_twq(const Lm& c, const uint64_t* lo, const uint64_t* hi, uint32_t s0) {
    using C = LmCfg<B>;
    for (uint32_t i = threadIdx.x; i < C::SEQS * C::N; i += LM_THREADS)
        at64(c.sm + C::O_TWQ + 8 * i) = gl_to_mont(tw2g(lo, hi, (s0 + i % C::SEQS) * (i / C::SEQS)));
}

// A CTA's share of blocks x columns, in units of one block and up to `width`
// columns (the block's tables are made once per unit): unit(block), then
// column(col) for each, the groups taking turns.
template <int B, class U, class F>
__device__ __forceinline__ void for_units(const Lm& c, uint32_t blocks, uint32_t cols, uint32_t width, U&& unit,
                                          F&& column) {
    const uint32_t per = (cols + width - 1) / width;
    for (uint32_t u = blockIdx.x; u < blocks * per; u += gridDim.x) {
        __syncthreads();  // the tables' last use
        unit(u / per);
        __syncthreads();
        const uint32_t c0 = (u % per) * width, c1 = c0 + width < cols ? c0 + width : cols;
        for (uint32_t col = c0 + c.group; col < c1; col += LmCfg<B>::GROUPS) column(u / per, col);
    }
}

// First round: this thread's outputs k = 8 * part + i of line (t, d), times
// table[d * TWP + k], become word d of the lines t + SEQS * k of the second
// round.  Of those lines' numbers only the bit 2 of SEQS * i changes the swizzle,
// so two base addresses serve all eight.
template <int B>
__device__ __forceinline__ void lm_round1(Lm& c, uint32_t t, uint32_t d, const uint8_t* table) {
    using C = LmCfg<B>;
    const uint64_t* tw = reinterpret_cast<const uint64_t*>(table) + d * C::TWP + 8 * c.part;
    uint8_t* dst[2];
#pragma unroll
    for (int i = 0; i < 2; i++) dst[i] = c.a + a_word<B>(t + C::SEQS * (8 * c.part + i), d) - 128 * C::SEQS * i;
    lm_dft<B>(c, [&](int i, uint64_t x) { at64(dst[i & 1] + 128 * C::SEQS * i) = gl_mont_mul(x, tw[i]); });
}

}  // namespace

// K1, and pass A of the plain NTT: Y[i1 + n1*k] = w^(i1 k) * (DFT over i2 of
// in[i1 + n1*i2])[k], n1 = 2^l1, R*R points; wlo, whi hold powers of w = w_N^-1 or
// w_N.  INV: the inverse DFT, taken as the forward one of the index-negated
// sequence (ntt.cu, k_lde_inv_a and k_pass_a).
template <int B, bool INV>
__global__ void __launch_bounds__(LM_THREADS, 1) k_pass_a_mma(const uint64_t* __restrict__ in, uint64_t ild,
                                                              uint64_t* __restrict__ Y, uint64_t yld, uint32_t cols,
                                                              uint32_t unit, int l1, const uint64_t* tw12, const uint64_t* wlo,
                                                              const uint64_t* whi, uint64_t* status) {
    using C = LmCfg<B>;
    Lm c;
    lm_init<B>(c, tw12);
    const uint32_t t = c.row % C::SEQS, d = c.row / C::SEQS;
    const uint64_t* twq = reinterpret_cast<const uint64_t*>(c.sm + C::O_TWQ) + 1024 * c.part + c.row;
    for_units<B>(
        c, (1u << l1) / C::SEQS, cols, unit, [&](uint32_t block) { fill_twq<B>(c, wlo, whi, C::SEQS * block); },
        [&](uint32_t block, uint32_t col) {
            const uint64_t* src = in + col * ild + C::SEQS * block + t;
            uint64_t* dst = Y + col * yld + C::SEQS * block + t;
            uint64_t v[8];
            lm_load<B, INV>(v, src, d + C::R * 8 * c.part, l1);
            lm_fill<B>(c, v);
            lm_round1<B>(c, t, d, c.sm + C::O_TW);
            dst += (uint64_t)(8 * C::R * c.part + d) << l1;
            lm_store<B>(c, dst, l1, [&](int i, uint64_t x) { return gl_mont_mul(x, twq[128 * i]); });
        });
    lm_done<B>(c, status);
}

// K2: rows k2 of Y (R*R points): inverse DFT -> coefficients; per coset c: times
// N^-1 s_c^i, forward DFT, times w_N^(k2 q) -> Z_c[k2 + n2*q], n2 = 2^l2.  The
// coset scale is applied as in k_lde_mid_sym2: s_c^(n2*ln) rides on the first
// round's output twiddle (one table per coset), the rest is one product with a
// table entry per (row, k1) of the block.  RAND: the raw coefficients i < rm get
// the addends of launch_rand_addend first.
template <int B, bool RAND>
__global__ void __launch_bounds__(LM_THREADS, 1) k_lde_mid_mma(const uint64_t* __restrict__ Y, uint64_t yld,
                                                               uint64_t* __restrict__ Z, uint32_t cols, uint32_t unit,
                                                               int l2, int le,
                                                               const uint64_t* tw12, const uint64_t* wlo,
                                                               const uint64_t* whi, const uint64_t* sc_lo,
                                                               const uint64_t* sc_hi, int hi_len,
                                                               const uint64_t* __restrict__ add, int rm,
                                                               uint64_t* status) {
    using C = LmCfg<B>;
    Lm c;
    lm_init<B>(c, tw12);
    const int E = 1 << le;
    const uint64_t N = (uint64_t)C::N << l2;
    uint8_t *scl = c.sm + C::O_SCL, *twc = scl + E * C::SCL_BYTES;
    for (uint32_t i = threadIdx.x; i < (uint32_t)E * C::N; i += LM_THREADS) {  // w^(d k) s_c^(n2 d)
        const uint32_t e = i / C::N, dd = i / C::R % C::R, k = i % C::R;
        const uint64_t s = gl_to_mont(gl_mul(tw2g(sc_lo + 4096 * e, sc_hi + hi_len * e, dd << l2), N));
        at64(twc + e * C::TWC_BYTES + 8 * (dd * C::TWP + k)) =
            gl_mont_mul(gl_to_mont(__ldg(tw12 + (4096 / C::N) * dd * k)), s);
    }
    const uint32_t t = c.row % C::SEQS, d = c.row / C::SEQS;  // lines t + SEQS * d
    const uint32_t tr = c.row / C::R, dr = c.row % C::R;      // lines d + R * t (rows read from memory)
    const uint64_t* twq = reinterpret_cast<const uint64_t*>(c.sm + C::O_TWQ) + 1024 * c.part + c.row;
    for_units<B>(
        c, (1u << l2) / C::SEQS, cols, unit,
        [&](uint32_t block) {
            const uint32_t k20 = C::SEQS * block;
            fill_twq<B>(c, wlo, whi, k20);
            for (uint32_t i = threadIdx.x; i < (uint32_t)E * LM_LINES; i += LM_THREADS) {  // N^-1 s_c^(k2 + R n2 k1)
                const uint32_t e = i / LM_LINES, tt = i % LM_LINES / C::R, k1 = i % C::R;
                const uint64_t *lo = sc_lo + 4096 * e, *hi = sc_hi + hi_len * e;  // sc_hi carries N^-1
                at64(scl + e * C::SCL_BYTES + 8 * (tt * C::TWP + k1)) =
                    gl_to_mont(gl_mul(gl_mul(tw2g(lo, hi, k20 + tt), tw2g(lo, hi, k1 << (B + l2))), N));
            }
        },
        [&](uint32_t block, uint32_t col) {
            const uint32_t k20 = C::SEQS * block;
            const uint64_t* src = Y + col * yld + (uint64_t)(k20 + tr) * C::N;
            uint64_t cf[8];
            lm_load<B, true>(cf, src, dr + C::R * 8 * c.part, 0);
            lm_fill<B>(c, cf);
            lm_round1<B>(c, tr, dr, c.sm + C::O_TW);
            // coefficients c[R * k1 + d] of row k20 + t, k1 = 8 * part + i
            lm_dft<B>(c, [&](int i, uint64_t x) { cf[i] = x; });
            uint64_t* dst = Z + (uint64_t)col * E * N + k20 + t + ((uint64_t)(8 * C::R * c.part + d) << l2);
#pragma unroll 1
            for (int e = 0; e < E; e++, dst += N) {
                const uint64_t* sc = reinterpret_cast<const uint64_t*>(scl + e * C::SCL_BYTES) + t * C::TWP + 8 * c.part;
                uint64_t v[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    uint64_t x = cf[i];
                    if constexpr (RAND) {  // addends of the first rm coefficients
                        const uint32_t ci = ((uint32_t)(C::R * (8 * c.part + i) + d) << l2) + k20 + t;
                        if (ci < (uint32_t)rm) x = gl_add_pc(x, add[((uint64_t)col * E + e) * rm + ci]);
                    }
                    v[i] = gl_mont_mul(x, sc[i]);
                }
                lm_fill<B>(c, v);
                lm_round1<B>(c, t, d, twc + e * C::TWC_BYTES);
                lm_store<B>(c, dst, l2, [&](int i, uint64_t x) { return gl_mont_mul(x, twq[128 * i]); });
            }
        });
    lm_done<B>(c, status);
}

// K3, and pass B of the plain NTT: rows of R*R points, forward DFT (INV: inverse,
// by negated index), written interleaved: out[E*(n1*q + q2) + c], n1 = 2^l1 rows
// q2 per coset, E = 2^le cosets; with INV each output times `scale` (Montgomery form).  Sequence u = E*q2 + c; a tile takes SEQS consecutive ones.
template <int B, bool INV>
__global__ void __launch_bounds__(LM_THREADS, 1) k_pass_b_mma(const uint64_t* __restrict__ Z,
                                                              uint64_t* __restrict__ out, uint64_t old, uint32_t cols,
                                                              int l1, int le, const uint64_t* tw12, uint64_t scale,
                                                              uint64_t* status) {
    using C = LmCfg<B>;
    Lm c;
    lm_init<B>(c, tw12);
    const uint32_t t = c.row % C::SEQS, d = c.row / C::SEQS;
    const uint32_t tr = c.row / C::R, dr = c.row % C::R;
    const uint32_t lb = l1 + le - (7 - B);  // log2 of the tiles per column
    const uint64_t tiles = (uint64_t)cols << lb, step = (uint64_t)gridDim.x * C::GROUPS;
    uint64_t v[8];
    auto load = [&](uint64_t tile) {
        const uint64_t col = tile >> lb;
        const uint32_t u = C::SEQS * (uint32_t)(tile & ((1u << lb) - 1)) + tr;
        const uint64_t* src = Z + (col << (l1 + 2 * B + le)) + ((uint64_t)(u & ((1u << le) - 1)) << (l1 + 2 * B)) +
                              ((uint64_t)(u >> le) << (2 * B));
        lm_load<B, INV>(v, src, dr + C::R * 8 * c.part, 0);
    };
    uint64_t tile = (uint64_t)blockIdx.x * C::GROUPS + c.group;
    if (tile < tiles) load(tile);
    for (; tile < tiles; tile += step) {
        lm_fill<B>(c, v);
        if (tile + step < tiles) load(tile + step);  // in flight during this tile's rounds
        lm_round1<B>(c, tr, dr, c.sm + C::O_TW);
        uint64_t* dst = out + (tile >> lb) * old + C::SEQS * (tile & ((1u << lb) - 1)) + t +
                        ((uint64_t)(8 * C::R * c.part + d) << (l1 + le));
        lm_store<B>(c, dst, l1 + le, [&](int, uint64_t x) { return INV ? gl_mont_mul(x, scale) : x; });
    }
    lm_done<B>(c, status);
}

namespace {

int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return sms;
}

// kern(args..., status); at most one CTA per SM.
template <class... P, class... A>
cudaError_t launch(void (*kern)(P...), uint64_t work, uint32_t bytes, cudaStream_t st, uint64_t* status, A... args) {
    const cudaError_t e = raise_smem_limit((const void*)kern);
    if (e != cudaSuccess) return e;
    const uint64_t sms = (uint64_t)sm_count();
    count_launch();
    kern<<<(unsigned)(work < sms ? work : sms), LM_THREADS, bytes + LM_SLACK, st>>>(args..., status);
    return mma_launched(status, st);
}

// Columns per unit: sixteen, to share a block's tables widely, but fewer (down to
// one per group) while that leaves fewer than two units per SM.  Units are dealt
// whole, so that the busiest CTA can have up to 1.3 times the mean (K1 and K2 of 51
// columns of 2^20: 1.27; of 379 columns of 2^16: 1.17).
template <int B>
uint32_t unit_cols(uint64_t blocks, uint32_t cols) {
    uint32_t unit = 16;
    while (unit > (uint32_t)LmCfg<B>::GROUPS && blocks * ((cols + unit - 1) / unit) < 2 * (uint64_t)sm_count()) unit /= 2;
    return unit;
}

template <int B>
cudaError_t pass_a(const LdePlan& pl, bool inverse, const uint64_t* in, uint64_t ild, uint64_t* Y, uint64_t yld,
                   uint32_t cols, int l1, cudaStream_t st, uint64_t* status) {
    using C = LmCfg<B>;
    const uint64_t blocks = (1u << l1) / C::SEQS;
    const uint32_t unit = unit_cols<B>(blocks, cols);
    return launch(inverse ? k_pass_a_mma<B, true> : k_pass_a_mma<B, false>, blocks * ((cols + unit - 1) / unit),
                  C::BYTES, st, status, in, ild, Y, yld, cols, unit, l1, pl.tw12_f, inverse ? pl.wn_i_lo : pl.wn_f_lo,
                  inverse ? pl.wn_i_hi : pl.wn_f_hi);
}
template <int B>
cudaError_t mid(const LdePlan& pl, const uint64_t* Y, uint64_t yld, uint64_t* Z, uint32_t cols, int l2, int hi_len,
                const uint64_t* add, int rm, cudaStream_t st, uint64_t* status) {
    using C = LmCfg<B>;
    const uint64_t blocks = (1u << l2) / C::SEQS;
    const uint32_t unit = unit_cols<B>(blocks, cols);
    return launch(rm ? k_lde_mid_mma<B, true> : k_lde_mid_mma<B, false>, blocks * ((cols + unit - 1) / unit),
                  C::mid_bytes(pl.log_exp), st, status, Y, yld, Z, cols, unit, l2, pl.log_exp, pl.tw12_f, pl.wn_f_lo,
                  pl.wn_f_hi, pl.sc_lo, pl.sc_hi, hi_len, add, rm);
}
template <int B>
cudaError_t pass_b(const LdePlan& pl, bool inverse, const uint64_t* Z, uint64_t* out, uint64_t old, uint32_t cols,
                   int l1, int le, uint64_t scale, cudaStream_t st, uint64_t* status) {
    using C = LmCfg<B>;
    const uint64_t tiles = ((uint64_t)cols << (l1 + le)) / C::SEQS;
    return launch(inverse ? k_pass_b_mma<B, true> : k_pass_b_mma<B, false>, (tiles + C::GROUPS - 1) / C::GROUPS,
                  C::BYTES, st, status, Z, out, old, cols, l1, le, pl.tw12_f, scale);
}

}  // namespace

cudaError_t launch_pass_a_mma(int lsub, const LdePlan& pl, bool inverse, const uint64_t* in, uint64_t ild, uint64_t* Y,
                              uint64_t yld, uint32_t cols, int l1, cudaStream_t st, uint64_t* status) {
    return lsub == 10 ? pass_a<5>(pl, inverse, in, ild, Y, yld, cols, l1, st, status)
                      : pass_a<4>(pl, inverse, in, ild, Y, yld, cols, l1, st, status);
}

cudaError_t launch_lde_mid_mma(int lsub, const LdePlan& pl, const uint64_t* Y, uint64_t yld, uint64_t* Z, uint32_t cols,
                               int l2, int hi_len, const uint64_t* add, int rm, cudaStream_t st, uint64_t* status) {
    return lsub == 10 ? mid<5>(pl, Y, yld, Z, cols, l2, hi_len, add, rm, st, status)
                      : mid<4>(pl, Y, yld, Z, cols, l2, hi_len, add, rm, st, status);
}

cudaError_t launch_pass_b_mma(int lsub, const LdePlan& pl, bool inverse, const uint64_t* Z, uint64_t* out, uint64_t old,
                              uint32_t cols, int l1, int le, uint64_t scale_mont, cudaStream_t st, uint64_t* status) {
    return lsub == 10 ? pass_b<5>(pl, inverse, Z, out, old, cols, l1, le, scale_mont, st, status)
                      : pass_b<4>(pl, inverse, Z, out, old, cols, l1, le, scale_mont, st, status);
}

unsigned int lde_mma_timeouts() {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_mma8_timeouts, sizeof v);
    return v;
}

}  // namespace tvmc
