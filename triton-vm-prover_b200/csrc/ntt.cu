// Batched Goldilocks NTT and fused low-degree extension (sm_100a).
//
// Every transform here is the DFT X[k] = sum_i x[i] w^(ik) with natural-order
// input and output, w = 7^((p-1)/n) (src/types/b_field_element.cpp:179-192);
// the inverse uses w^-1 and scales by n^-1 (src/ntt/ntt.cpp:59-86).  Results
// are canonical, so they equal the reference's radix-2 DIT bit for bit.
//
// Global structure.  Sizes up to 2^11 run in one pass per column (whole column
// in one CTA).  Larger sizes use the four-step split n = n1*n2, i = i1 + n1*i2,
// k = n2*k1 + k2:
//   pass A: for each i1, DFT_n2 over i2 (elements at stride n1), times w^(i1*k2)
//   pass B: for each k2, DFT_n1 over i1 (contiguous rows) -> X[n2*k1 + k2]
// A CTA moves T sequences at a time so that global accesses come in runs of T
// consecutive words.
//
// In-CTA structure (sub_dft).  A sub-transform of size 2^LS <= 2^12 is itself
// split four-step into rounds of radix <= 32: in each round a thread holds one
// line of R elements in registers and runs a radix-2 DIF network on it.  The
// first round takes its inputs straight from a load function (global memory,
// or shared memory times a scale) and the last round hands its outputs to a
// store function (global memory times a twiddle), so shared memory carries only
// the transposes between rounds: one write and one read per element per
// round boundary, one barrier per boundary.
//
// LDE (LDE::extend_column, src/ntt/ntt.cpp:121-131; evaluate_on_coset :94-117):
// the E*N-point forward transform of the zero-padded, offset-scaled
// coefficients is evaluated as E cosets of size N, LDE[E*q + c] =
// DFT_N(coef_i * s_c^i)[q] with s_c = offset * w_{EN}^c, because
// w_{EN}^(i(Eq+c)) = w_N^(iq) * w_{EN}^(ic).  The inverse's pass B and the
// forward's pass A touch the same index sets when the forward split is taken
// as (n2, n1), so one kernel does both for all E cosets:
//   K1 (lde_inv_a): inverse pass A, trace -> Y
//   K2 (lde_mid):   inverse pass B, scale by N^-1 s_c^i, forward pass A -> Z_c
//   K3 (lde_fwd_b): forward pass B for all cosets, written interleaved -> LDE
#include <algorithm>

#include "internal.cuh"
#include "field.cuh"
#include "lde_mma.h"
#include "ntt_sub.cuh"

namespace tvmc {

// The forward 32-point root as a power of two, as the register networks apply it.
constexpr int GL_W32_LOG2 = 78;
static_assert(GL_W32_LOG2 == W32_LOG2, "the networks of ntt_sub.cuh use this root");

// ---------------------------------------------------------------- plain NTT

// Whole columns per CTA: T = 2^lT columns, size 2^LS <= 2^11, in place.  All
// transforms run on the forward root (tw12 = w_4096 powers); INV negates the
// input index, which turns the forward DFT into the inverse one (reg_dft).
template <int LS, bool INV>
__global__ void __launch_bounds__(NTT_THREADS) k_ntt_small(uint64_t* data, uint64_t ld, uint64_t cols, int lT,
                                                           const uint64_t* tw12, uint64_t scale) {
    extern __shared__ uint64_t sm[];
    uint64_t* tw = sm;
    uint64_t* s = sm + (1 << LS);
    load_tw<LS>(tw, tw12);
    __syncthreads();
    const uint64_t c0 = (uint64_t)blockIdx.x << lT;
    constexpr int nm = (1 << LS) - 1;
    sub_dft<LS>(
        s, lT, tw,
        [&](int k, int t) { return c0 + t < cols ? gl_canon(data[(c0 + t) * ld + (INV ? -k & nm : k)]) : 0ull; },
        [&](int k, int t, uint64_t v) {
            if (c0 + t < cols) data[(c0 + t) * ld + k] = gl_mul_c(v, scale);
        });
}

// Pass A: out[i1 + n1*k2] = w^(i1*k2) * DFT_n2(in[i1 + n1*i2])[k2]; in may equal out.
// tw12 is the forward table; INV: inverse sub-DFT (negated input index).
template <int L2, bool INV>
__global__ void __launch_bounds__(NTT_THREADS) k_pass_a(const uint64_t* in, uint64_t ild, uint64_t* out,
                                                        uint64_t old, int l1, int lT, const uint64_t* tw12,
                                                        const uint64_t* wlo, const uint64_t* whi) {
    extern __shared__ uint64_t sm[];
    uint64_t* tw = sm;
    uint64_t* s = sm + (1 << L2);
    load_tw<L2>(tw, tw12);
    __syncthreads();
    const uint32_t i10 = blockIdx.x << lT;
    const uint64_t* src = in + (uint64_t)blockIdx.y * ild + i10;
    uint64_t* dst = out + (uint64_t)blockIdx.y * old + i10;
    constexpr int n2m = (1 << L2) - 1;
    sub_dft<L2, true>(
        s, lT, tw, [&](int k, int t) { return gl_canon(src[t + ((uint64_t)(INV ? -k & n2m : k) << l1)]); },
        [](int, int, uint64_t) {});
    __syncthreads();
    const int T = 1 << lT;
    for (int idx = threadIdx.x; idx < (T << L2); idx += blockDim.x) {
        const int t = idx & (T - 1), k2 = idx >> lT;
        const uint64_t v = s[spos(out_pos<L2>(k2), lT) + t];
        dst[t + ((uint64_t)k2 << l1)] = gl_mul_c(v, tw2(wlo, whi, (i10 + t) * (uint32_t)k2));
    }
}

// Pass B: out[n2*k1 + k2] = scale * DFT_n1(in[i1 + n1*k2])[k1]; in != out.
// tw12 is the forward table; INV: inverse sub-DFT (negated input index).
template <int L1, bool INV>
__global__ void __launch_bounds__(NTT_THREADS) k_pass_b(const uint64_t* in, uint64_t ild, uint64_t* out,
                                                        uint64_t old, int l2, int lT, const uint64_t* tw12,
                                                        uint64_t scale) {
    extern __shared__ uint64_t sm[];
    uint64_t* tw = sm;
    uint64_t* s = sm + (1 << L1);
    load_tw<L1>(tw, tw12);
    __syncthreads();
    const uint32_t k20 = blockIdx.x << lT;
    const uint64_t* src = in + (uint64_t)blockIdx.y * ild + ((uint64_t)k20 << L1);
    uint64_t* dst = out + (uint64_t)blockIdx.y * old + k20;
    constexpr int n1m = (1 << L1) - 1;
    sub_dft<L1>(
        s, lT, tw, [&](int k, int t) { return src[((uint64_t)t << L1) + (INV ? -k & n1m : k)]; },
        [&](int k, int t, uint64_t v) { dst[((uint64_t)k << l2) + t] = gl_mul_c(v, scale); });
}

// ---------------------------------------------------------------------- LDE

// K1: inverse pass A over the trace: Y[i1 + n1*k2] = w^-(i1*k2) DFT^-1_n2(...)[k2],
// the inverse DFT taken as the forward one of the index-negated column (reg_dft).
// At 2^10-point passes the unbounded allocation takes 136 registers (one
// 256-thread CTA per SM); capping it at two CTAs per SM is 4% faster on the
// 2^20-row LDE.  The other kernels keep their unbounded allocations, which
// measured faster than capped ones.
template <int L2>
__global__ void __launch_bounds__(NTT_THREADS, L2 == 10 ? 2 : 1) k_lde_inv_a(const uint64_t* trace, uint64_t tld, uint64_t* Y,
                                                           uint64_t yld, int l1, int lT, const uint64_t* tw12_f,
                                                           const uint64_t* wlo, const uint64_t* whi) {
    extern __shared__ uint64_t sm[];
    uint64_t* tw = sm;
    uint64_t* s = sm + (1 << L2);
    load_tw<L2, true>(tw, tw12_f);
    __syncthreads();
    const uint32_t i10 = blockIdx.x << lT;
    const uint64_t* src = trace + (uint64_t)blockIdx.y * tld + i10;
    uint64_t* dst = Y + (uint64_t)blockIdx.y * yld + i10;
    constexpr int n2m = (1 << L2) - 1;
    // offsets within a column are below N <= 2^22: 32-bit index arithmetic
    sub_dft<L2, true, true>(
        s, lT, tw, [&](int k, int t) { return gl_canon(src[(uint32_t)t + ((uint32_t)(-k & n2m) << l1)]); },
        [](int, int, uint64_t) {});
    __syncthreads();
    const int T = 1 << lT;
    for (int idx = threadIdx.x; idx < (T << L2); idx += blockDim.x) {
        const int t = idx & (T - 1), k2 = idx >> lT;
        const uint64_t v = s[spos(out_pos<L2>(k2), lT) + t];
        dst[(uint32_t)t + ((uint32_t)k2 << l1)] = gl_mul_c(v, tw2(wlo, whi, (i10 + t) * (uint32_t)k2));
    }
}

// K2: rows k2 in [k20, k20+T) of Y: inverse DFT_n1 -> coefficients c[n2*k1 + k2];
// per coset: a = c * N^-1 s_c^i, forward DFT_n1 over k1, times w_N^(k2*q2),
// Z_c[k2 + n2*q2].  Z holds E planes of N words per column: Z[(col*E + c)*N + .].
template <int L1, bool RAND>
__global__ void __launch_bounds__(NTT_THREADS) k_lde_mid(const uint64_t* Y, uint64_t yld, uint64_t* Z, int l2,
                                                         int lT, int le, const uint64_t* tw12_f, const uint64_t* wlo,
                                                         const uint64_t* whi, const uint64_t* sc_lo,
                                                         const uint64_t* sc_hi, int hi_len, const uint64_t* add,
                                                         int rm) {
    extern __shared__ uint64_t sm[];
    constexpr int n1 = 1 << L1;
    const int E = 1 << le;
    uint64_t* twf = sm;  // forward root only (the inverse negates its input index)
    uint64_t* cf = twf + n1;                 // coefficients, natural k1 order
    uint64_t* s = cf + spad_words(n1, lT);   // transposes
    load_tw<L1>(twf, tw12_f);
    __syncthreads();
    const uint64_t col = blockIdx.y;
    const uint32_t k20 = blockIdx.x << lT;
    const uint64_t* src = Y + col * yld + ((uint64_t)k20 << L1);
    sub_dft<L1>(  // inverse: forward DFT of the index-negated row
        s, lT, twf, [&](int k, int t) { return src[((uint64_t)t << L1) + (-k & (n1 - 1))]; },
        [&](int k, int t, uint64_t v) { cf[spos(k, lT) + t] = v; });
    __syncthreads();
    const uint64_t N = 1ull << (L1 + l2);
    for (int c = 0; c < E; c++) {
        const uint64_t* lo = sc_lo + 4096 * c;
        const uint64_t* hi = sc_hi + hi_len * c;
        uint64_t* dst = Z + (col * E + c) * N + k20;
        sub_dft<L1, true>(
            s, lT, twf,
            [&](int k, int t) {
                uint64_t x = cf[spos(k, lT) + t];
                const uint32_t i = ((uint32_t)k << l2) + k20 + t;
                if constexpr (RAND) {
                    if (i < (uint32_t)rm) x = gl_add_pc(x, add[(col * E + c) * rm + i]);
                }
                return gl_mul_c(x, tw2(lo, hi, i));
            },
            [](int, int, uint64_t) {});
        __syncthreads();
        const int T = 1 << lT;
        for (int idx = threadIdx.x; idx < (T << L1); idx += blockDim.x) {
            const int t = idx & (T - 1), q = idx >> lT;
            const uint64_t v = s[spos(out_pos<L1>(q), lT) + t];
            dst[t + ((uint64_t)q << l2)] = gl_mul_c(v, tw2(wlo, whi, (k20 + t) * (uint32_t)q));
        }
        __syncthreads();
    }
}

// K2 for two-round sub-transforms (n1 <= 2^10), 128 threads = T lines x R2.
// The inverse DFT_n1 ends with thread (t, k) holding coefficients
// c[R2*k1 + k], k1 < R1, in registers; splitting the forward DFT_n1 as
// i = i1 + R2*i2 makes its first round take exactly that set (i1 = k), so the
// coefficients stay in registers for all E cosets and only the forward's
// second round goes through shared memory.
template <int L1, bool RAND>
__global__ void __launch_bounds__(128) k_lde_mid_reg(const uint64_t* Y, uint64_t yld, uint64_t* Z, int l2, int le,
                                                     const uint64_t* tw12_f,
                                                     const uint64_t* wlo, const uint64_t* whi,
                                                     const uint64_t* sc_lo, const uint64_t* sc_hi, int hi_len,
                                                     const uint64_t* add, int rm) {
    using PL = Plan<L1>;
    static_assert(PL::NR == 2, "two-round sizes only");
    constexpr int b1 = PL::b1, b2 = PL::b2, R1 = 1 << b1, R2 = 1 << b2;
    constexpr int lT = 7 - b2, T = 1 << lT;  // T * R2 = 128 threads
    constexpr int n1 = 1 << L1;
    extern __shared__ uint64_t sm[];
    uint64_t* twf = sm;  // forward root only (the inverse negates its input index)
    uint64_t* s = twf + n1;
    load_tw<L1>(twf, tw12_f);
    __syncthreads();
    const int E = 1 << le;
    const uint64_t col = blockIdx.y;
    const uint32_t k20 = blockIdx.x << lT;
    const uint64_t* src = Y + col * yld + ((uint64_t)k20 << L1);
    // inverse, round 1: digit 2 (stride R1), lines (t, d1)
    for (int id = threadIdx.x; id < (R1 << lT); id += blockDim.x) {
        const int t = id & (T - 1), d1 = id >> lT;
        uint64_t v[R2];
#pragma unroll
        for (int j = 0; j < R2; j++) v[j] = src[((uint64_t)t << L1) + (-(d1 + (j << b1)) & (n1 - 1))];
        reg_dft<b2>(v);  // inverse as the forward DFT of the index-negated row
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            uint64_t x = v[brevc<b2>(k2)];
            if (k2) x = gl_mul_c(x, twf[d1 * k2]);
            s[spos2<b1>(d1, k2, lT) + t] = x;
        }
    }
    __syncthreads();
    // inverse, round 2: this thread's line (t, kk) -> c[R2*k1 + kk]
    const int t = threadIdx.x & (T - 1), kk = threadIdx.x >> lT;
    uint64_t cf[R1];
    {
        uint64_t v[R1];
#pragma unroll
        for (int d1 = 0; d1 < R1; d1++) v[d1] = s[spos(d1 + (kk << b1), lT) + t];
        reg_dft<b1>(v);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) cf[k1] = v[brevc<b1>(k1)];
    }
    __syncthreads();
    const uint64_t N = 1ull << (L1 + l2);
    for (int c = 0; c < E; c++) {
        const uint64_t* lo = sc_lo + 4096 * c;
        const uint64_t* hi = sc_hi + hi_len * c;
        // forward, round 1 on the register line: a[kk + R2*i2] * N^-1 s_c^i, DFT over i2
        {
            uint64_t v[R1];
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) {
                const uint32_t ci = (uint32_t)kk + ((uint32_t)k1 << b2);
                const uint32_t i = (ci << l2) + k20 + t;
                uint64_t x = cf[k1];
                if constexpr (RAND) {
                    if (i < (uint32_t)rm) x = gl_add_pc(x, add[(col * E + c) * rm + i]);
                }
                v[k1] = gl_mul_c(x, tw2(lo, hi, i));
            }
            reg_dft<b1>(v);
#pragma unroll
            for (int q = 0; q < R1; q++) {
                uint64_t x = v[brevc<b1>(q)];
                if (kk * q) x = gl_mul_c(x, twf[kk * q]);
                s[spos(kk + (q << b2), lT) + t] = x;
            }
        }
        __syncthreads();
        // forward, round 2: lines (t, q2), DFT over i1 -> X[R1*q1 + q2] at slot q1 + R2*q2
        for (int id = threadIdx.x; id < (R1 << lT); id += blockDim.x) {
            const int tt = id & (T - 1), q2 = id >> lT;
            uint64_t w[R2];
#pragma unroll
            for (int i1 = 0; i1 < R2; i1++) w[i1] = s[spos(i1 + (q2 << b2), lT) + tt];
            reg_dft<b2>(w);
#pragma unroll
            for (int q1 = 0; q1 < R2; q1++) s[spos(q1 + (q2 << b2), lT) + tt] = w[brevc<b2>(q1)];
        }
        __syncthreads();
        uint64_t* dst = Z + (col * E + c) * N + k20;
        for (int idx = threadIdx.x; idx < (T << L1); idx += blockDim.x) {
            const int tt = idx & (T - 1), q = idx >> lT;
            const uint64_t x = s[spos((q >> b1) + ((q & (R1 - 1)) << b2), lT) + tt];
            dst[tt + ((uint64_t)q << l2)] = gl_mul_c(x, tw2(wlo, whi, (k20 + tt) * (uint32_t)q));
        }
        __syncthreads();
    }
}

// K2 for n1 = R*R (2^6, 2^8, 2^10): as k_lde_mid_reg, but the inverse and the
// E forward transforms run through ONE rolled loop over (pass, round) around
// a single register DFT body, so the kernel's code stays small enough for the
// instruction cache.  Thread (t, ln) owns line ln of every round.
template <int L1, int MINB, bool RAND>
__global__ void __launch_bounds__(128, MINB) k_lde_mid_sym(const uint64_t* Y, uint64_t yld, uint64_t* Z, int l2, int le,
                                                     const uint64_t* tw12_f,
                                                     const uint64_t* wlo, const uint64_t* whi,
                                                     const uint64_t* sc_lo, const uint64_t* sc_hi, int hi_len,
                                                     const uint64_t* add, int rm) {
    using PL = Plan<L1>;
    static_assert(PL::NR == 2 && PL::b1 == PL::b2, "square sizes only");
    constexpr int B = PL::b1, R = 1 << B;
    constexpr int lT = 7 - B, T = 1 << lT;  // T * R = 128 threads
    constexpr int n1 = 1 << L1;
    extern __shared__ uint64_t sm[];
    uint64_t* twf = sm;  // forward root only (the inverse negates its input index)
    uint64_t* s = twf + n1;
    load_tw<L1>(twf, tw12_f);
    __syncthreads();
    const int E = 1 << le;
    const uint64_t col = blockIdx.y;
    const uint32_t k20 = blockIdx.x << lT;
    const uint64_t* src = Y + col * yld + ((uint64_t)k20 << L1);
    const uint64_t N = 1ull << (L1 + l2);
    const int t = threadIdx.x & (T - 1), ln = threadIdx.x >> lT;
    uint64_t cf[R];  // coefficients c[R*k1 + ln] of row k20 + t
#pragma unroll 1
    for (int pass = 0; pass <= E; pass++) {  // 0: inverse; c + 1: forward, coset c
        const uint64_t* tw = twf;  // the inverse runs forward on the index-negated row
        const uint64_t* lo = sc_lo + 4096 * (pass ? pass - 1 : 0);
        const uint64_t* hi = sc_hi + hi_len * (pass ? pass - 1 : 0);
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            uint64_t v[R];
            if (half == 0) {
                if (pass == 0) {  // inverse round 1: elements -(ln + R*j) of row t
#pragma unroll
                    for (int j = 0; j < R; j++) v[j] = src[((uint64_t)t << L1) + (-(ln + (j << B)) & (n1 - 1))];
                } else {  // forward round 1: c[ln + R*k1] * N^-1 s_c^i
#pragma unroll
                    for (int k1 = 0; k1 < R; k1++) {
                        const uint32_t ci = (uint32_t)ln + ((uint32_t)k1 << B);
                        const uint32_t i = (ci << l2) + k20 + t;
                        uint64_t x = cf[k1];
                        if constexpr (RAND) {
                            if (i < (uint32_t)rm) x = gl_add_pc(x, add[(col * E + pass - 1) * rm + i]);
                        }
                        v[k1] = gl_mul_c(x, tw2(lo, hi, i));
                    }
                }
            } else {  // round 2 of either: slots x + R*ln
#pragma unroll
                for (int x = 0; x < R; x++) v[x] = s[spos2<B>(x, ln, lT) + t];
            }
            reg_dft<B>(v);
            if (half == 0) {  // twiddle w^(ln*k), slot ln + R*k
#pragma unroll
                for (int k = 0; k < R; k++) {
                    uint64_t x = v[brevc<B>(k)];
                    if (ln * k) x = gl_mul_c(x, tw[ln * k]);
                    s[spos2<B>(ln, k, lT) + t] = x;
                }
            } else if (pass == 0) {
#pragma unroll
                for (int k1 = 0; k1 < R; k1++) cf[k1] = v[brevc<B>(k1)];
            } else {  // X[R*q1 + ln] stays in slot q1 + R*ln
#pragma unroll
                for (int q1 = 0; q1 < R; q1++) s[spos2<B>(q1, ln, lT) + t] = v[brevc<B>(q1)];
            }
            __syncthreads();
        }
        if (pass) {
            uint64_t* dst = Z + (col * E + pass - 1) * N + k20;
            for (int idx = threadIdx.x; idx < (T << L1); idx += blockDim.x) {
                const int tt = idx & (T - 1), q = idx >> lT;
                const uint64_t x = s[spos((q >> B) + ((q & (R - 1)) << B), lT) + tt];
                dst[tt + ((uint64_t)q << l2)] = gl_mul_c(x, tw2(wlo, whi, (k20 + tt) * (uint32_t)q));
            }
            __syncthreads();
        }
    }
}

// K2, table-sharing form of k_lde_mid_sym: the inter-pass twiddles
// w_N^(k2*q) are the same for all E cosets, so the CTA forms them once into
// shared memory (twq, T*n1 words) and every coset reads them there.  The coset
// scale N^-1 s_c^i, i = k2 + n2*ln + n2*R*k1, costs one product per element:
// s_c^(n2*ln) is constant over round 1's input index k1, so it rides on that
// round's output twiddle, whose per-coset table twf[ln][k] = w_n1^(ln*k)
// s_c^(n2*ln) the CTA refills before each coset; the rest comes from a
// per-coset table sbt[t][k1] = N^-1 s_c^(k2 + n2*R*k1).  All factors are in
// Montgomery form.  At n1 = 2^10 the CTA holds 74 KB of shared memory, so three
// CTAs still fit on an SM.
template <int L1, int MINB, bool RAND>
__global__ void __launch_bounds__(128, MINB) k_lde_mid_sym2(const uint64_t* Y, uint64_t yld, uint64_t* Z, int l2,
                                                            int le, const uint64_t* tw12_f, const uint64_t* wlo,
                                                            const uint64_t* whi, const uint64_t* sc_lo,
                                                            const uint64_t* sc_hi, int hi_len, const uint64_t* add,
                                                            int rm) {
    using PL = Plan<L1>;
    static_assert(PL::NR == 2 && PL::b1 == PL::b2, "square sizes only");
    constexpr int B = PL::b1, R = 1 << B;
    constexpr int lT = 7 - B, T = 1 << lT;  // T * R = 128 threads
    constexpr int n1 = 1 << L1;
    constexpr int RP = R + 1;  // padded table rows: the warp's lines (rows) fall in distinct banks
    extern __shared__ uint64_t sm[];
    uint64_t* twf = sm;                        // [ln*RP + k]: round-1 output twiddle of line ln, output k
    uint64_t* s = twf + R * RP;                // transposes
    uint64_t* twq = s + spad_words(n1, lT);    // w_N^((k20 + tt) * q) at [tt + T*q]
    uint64_t* sbt = twq + (T << L1);           // [t*RP + k1]: round-1 input scale of row t, element k1
    const int E = 1 << le;
    const uint64_t col = blockIdx.y;
    const uint32_t k20 = blockIdx.x << lT;
    const uint64_t N = 1ull << (L1 + l2);
    // twf holds w_n1^(ln*k) for the inverse and w_n1^(ln*k) * s_c^(n2*ln) for
    // coset c (Montgomery form): each thread fills KPT consecutive k of line bl,
    // forming the line factor bm once.
    constexpr int KPT = R * R >= 128 ? R * R / 128 : 1;
    const int bl = threadIdx.x / (R / KPT), bk = (threadIdx.x % (R / KPT)) * KPT;
    auto fill_twf = [&](uint64_t bm) {
        if (bl < R) {
#pragma unroll
            for (int j = 0; j < KPT; j++) {
                const int k = bk + j;
                const uint64_t w = __ldg(tw12_f + (((bl * k) & (n1 - 1)) << (12 - L1)));
                twf[bl * RP + k] = gl_mont_mul(gl_to_mont(w), bm);
            }
        }
    };
    fill_twf(0xFFFFFFFFull);  // 1 in Montgomery form
    for (int idx = threadIdx.x; idx < (T << L1); idx += blockDim.x)
        twq[idx] = gl_to_mont(tw2(wlo, whi, (k20 + (idx & (T - 1))) * (uint32_t)(idx >> lT)));
    __syncthreads();
    const uint64_t* src = Y + col * yld + ((uint64_t)k20 << L1);
    const int t = threadIdx.x & (T - 1), ln = threadIdx.x >> lT;
    const uint32_t i0 = ((uint32_t)ln << l2) + k20 + t;
    uint64_t cf[R];  // coefficients c[R*k1 + ln] of row k20 + t
#pragma unroll 1
    for (int pass = 0; pass <= E; pass++) {  // 0: inverse; c + 1: forward, coset c
        const int c = pass ? pass - 1 : 0;
        if (pass) {
            // the coset scale N^-1 s_c^i, i = k2 + n2*ln + n2*R*k1, k2 = k20 + t:
            // s_c^(n2*ln) is constant over round 1's input index k1, so it joins
            // that round's output twiddle (twf); the rest is one table entry per
            // (row t, element k1) (sbt).  tw2 on the scale tables carries N^-1.
            const uint64_t* lo = sc_lo + 4096 * c;
            const uint64_t* hi = sc_hi + hi_len * c;
            fill_twf(bl < R ? gl_to_mont(gl_mul(tw2(lo, hi, (uint32_t)bl << l2), N)) : 0);
            for (int idx = threadIdx.x; idx < T * R; idx += blockDim.x) {
                const int tt = idx >> B, k1 = idx & (R - 1);
                sbt[tt * RP + k1] = gl_to_mont(
                    gl_mul(gl_mul(tw2(lo, hi, k20 + tt), tw2(lo, hi, (uint32_t)k1 << (B + l2))), N));
            }
            __syncthreads();
        }
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            uint64_t v[R];
            if (half == 0) {
                if (pass == 0) {  // inverse round 1: elements -(ln + R*j) of row t
#pragma unroll
                    for (int j = 0; j < R; j++) v[j] = src[((uint64_t)t << L1) + (-(ln + (j << B)) & (n1 - 1))];
                } else {  // forward round 1: c[ln + R*k1] * N^-1 s_c^(k2 + n2*R*k1)
#pragma unroll
                    for (int k1 = 0; k1 < R; k1++) {
                        uint64_t x = cf[k1];
                        if constexpr (RAND) {
                            const uint32_t i = i0 + ((uint32_t)k1 << (B + l2));
                            if (i < (uint32_t)rm) x = gl_add_pc(x, add[(col * E + c) * rm + i]);
                        }
                        v[k1] = gl_mont_mul(x, sbt[t * RP + k1]);
                    }
                }
            } else {  // round 2 of either: slots x + R*ln
#pragma unroll
                for (int x = 0; x < R; x++) v[x] = s[spos2<B>(x, ln, lT) + t];
            }
            reg_dft<B>(v);
            if (half == 0) {  // twiddle twf[ln][k], slot ln + R*k
#pragma unroll
                for (int k = 0; k < R; k++) {
                    uint64_t x = v[brevc<B>(k)];
                    if (pass || ln * k) x = gl_mont_mul(x, twf[ln * RP + k]);
                    s[spos2<B>(ln, k, lT) + t] = x;
                }
            } else if (pass == 0) {
#pragma unroll
                for (int k1 = 0; k1 < R; k1++) cf[k1] = v[brevc<B>(k1)];
            } else {  // X[R*q1 + ln] stays in slot q1 + R*ln
#pragma unroll
                for (int q1 = 0; q1 < R; q1++) s[spos2<B>(q1, ln, lT) + t] = v[brevc<B>(q1)];
            }
            __syncthreads();
        }
        if (pass) {
            // thread (tt, q0) of the 128 = T x R stores X[q], q = q0 + R*m: its slot
            // is m + R*q0, its twiddle twq[threadIdx.x + 128*m], its address
            // dst + tt + (q0 << l2) + m*(R << l2) (bases hoisted out of the loop)
            const int tt = threadIdx.x & (T - 1), q0 = threadIdx.x >> lT;
            uint64_t* dst = Z + (col * E + c) * N + k20 + tt + ((uint64_t)q0 << l2);
            const uint64_t dstep = (uint64_t)R << l2;
            const uint64_t* twp = twq + threadIdx.x;
#pragma unroll 4
            for (int m = 0; m < R; m++) {
                const uint64_t x = s[spos2<B>(m, q0, lT) + tt];
                dst[m * dstep] = gl_mont_mul(x, twp[m << 7]);
            }
            __syncthreads();
        }
    }
}

// K3: for q2 in [q20, q20+T3), all E cosets: DFT_n2 over rows Z_c[i1' + n2*q2];
// E_c[n1*q1 + q2] -> LDE[E*(n1*q1 + q2) + c], written as runs of E*T3 words.
// Sequence u = E*t + c of the CTA is row q20 + t of coset c.
template <int L2>
__global__ void __launch_bounds__(NTT_THREADS) k_lde_fwd_b(const uint64_t* Z, uint64_t* out, uint64_t old,
                                                           int l1, int lT3, int le, const uint64_t* tw12_f) {
    extern __shared__ uint64_t sm[];
    const int E = 1 << le;
    const int lS = lT3 + le;
    uint64_t* tw = sm;
    uint64_t* s = sm + (1 << L2);
    load_tw<L2, true>(tw, tw12_f);
    __syncthreads();
    const uint64_t col = blockIdx.y;
    const uint32_t q20 = blockIdx.x << lT3;
    const uint64_t N = 1ull << (l1 + L2);
    const uint64_t* src = Z + col * E * N + ((uint64_t)q20 << L2);
    uint64_t* dst = out + col * old + (uint64_t)q20 * E;
    sub_dft<L2, false, true>(
        s, lS, tw,
        // offsets within a column are below E * N <= 2^26: 32-bit index arithmetic
        [&](int k, int u) {
            const uint32_t c = (uint32_t)u & (E - 1), t = (uint32_t)u >> le;
            return src[(c << (l1 + L2)) + (t << L2) + (uint32_t)k];
        },
        [&](int q, int u, uint64_t v) { dst[((uint32_t)q << (l1 + le)) + (uint32_t)u] = v; });
}

// N = 1: the interpolant is the constant trace value; coset c of the LDE is the
// single point s_c, where the randomizer term contributes add[(col*E + c)*rm].
__global__ void k_lde_one(const uint64_t* trace, uint64_t tld, uint64_t* out, uint64_t old, uint64_t total,
                          int le, const uint64_t* add, int rm) {
    const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const uint64_t col = idx >> le, c = idx & ((1u << le) - 1);
    uint64_t x = gl_canon(trace[col * tld]);
    if (rm) x = gl_add_c(x, add[idx * rm]);
    out[col * old + c] = x;
}

// Randomizer term of the zero-knowledge LDE, folded per coset into addends of
// the first rm = min(N, R) interpolant coefficients.  Per column the extended
// polynomial is a(x) + q(x) with q = (x^N - t^N) r(x), truncated to degree <
// qlen.  On coset c of the evaluation domain, x^N equals z_c = o^N w_E^c, so
// q(x) there equals sum_k z_c^k q_{i + kN} x^i (i < N).  The LDE kernels add
// out[(col*E + c)*rm + i] = N t^i sum_k z_c^k q_{i+kN} to the raw (unscaled)
// coefficient i before multiplying by N^-1 (s_c / t)^i.
__global__ void k_rand_addend(const uint64_t* r, uint64_t R, uint64_t total, int logn, int le, int rm, uint64_t t,
                              uint64_t tN, uint64_t oN, uint64_t wE, uint64_t qlen, uint64_t* out) {
    const uint64_t N = 1ull << logn;
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = idx % (uint64_t)rm, cc = idx / (uint64_t)rm;
        const uint64_t c = cc & ((1u << le) - 1), col = cc >> le;
        const uint64_t* rc = r + col * R;
        const uint64_t zc = gl_mul_c(oN, gl_canon(gl_pow(wE, c)));
        uint64_t acc = 0, zk = 1;
        for (uint64_t j = i; j < qlen; j += N) {
            uint64_t q = 0;
            if (j < R) q = gl_sub_c(0, gl_mul_c(tN, gl_canon(rc[j])));
            if (j >= N && j - N < R) q = gl_add_c(q, gl_canon(rc[j - N]));
            acc = gl_add_c(acc, gl_mul_c(zk, q));
            zk = gl_mul_c(zk, zc);
        }
        out[idx] = gl_mul_c(gl_mul_c(N % GL_P, gl_canon(gl_pow(t, i))), acc);
    }
}

cudaError_t launch_rand_addend(const uint64_t* r, uint64_t R, uint64_t cols, int logn, int le, uint64_t t,
                               uint64_t tN, uint64_t oN, uint64_t wE, uint64_t qlen, uint64_t* out, cudaStream_t st) {
    const int rm = rand_rows(logn, R);
    const uint64_t total = (cols << le) * (uint64_t)rm;
    if (total == 0) return cudaSuccess;
    const uint64_t blocks = (total + 255) / 256;
    count_launch();
    k_rand_addend<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, st>>>(r, R, total, logn, le, rm, t,
                                                                                   tN, oN, wE, qlen, out);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ helpers

static inline int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// T = 2^lT sequences so that T * 2^ls ~ 2^budget.  Sizes up to 2^5 run as one
// register round per sequence, so they take up to 256 sequences per CTA.
static int choose_lT(int ls, int budget_words_log) {
    return clampi(budget_words_log - ls, 0, ls <= 5 ? 8 : 3);
}

// The largest lT' <= lT whose tile fits in one CTA's shared memory: the
// 2^ls-word twiddle table plus nbuf transpose buffers of 2^(lT' + extra)
// sequences (extra: the E cosets K3 moves per sequence).
static int fit_lT(int lT, int ls, int nbuf, int extra = 0) {
    while (lT > 0 && ((size_t)(1u << ls) + (size_t)nbuf * spad_words(1 << ls, lT + extra)) * 8 > 227 * 1024) lT--;
    return lT;
}

// Whether the tensor-core passes pay for `cols` columns of 2^l points: they take
// one CTA per SM with tables of its own, so few short columns are better off on
// the register networks.  B200, us (networks | tensor cores): LDE x4 of 2^14 x 16
// 57 | 62, x 64 123 | 91, 2^15 x 16 73 | 76, x 64 201 | 173, 2^16 x 4 55 | 72, x 16 116 | 90,
// 2^17 x 1 90 | 49, 2^18 x 1 98 | 71, 2^20 x 1 150 | 151, x 64 6080 | 4298; inverse NTT of
// 2^14 x 64 34 | 36, x 256 92 | 79, 2^16 x 16 36 | 34, x 256 288 | 199, 2^18 x 4 34 | 42, x 16
// 101 | 84, 2^20 x 1 44 | 57, x 4 106 | 104.  An NTT of 2^22 points, whose splits
// leave one of its passes to networks of 2^11 or 2^12 points, does not gain: x 1
// 124 | 131, x 4 428 | 454, x 16 1665 | 1705; beyond it no pass has a tensor-core size.
static bool lde_mma_pays(int l, uint64_t cols) { return l >= 17 || (cols << l) >= 1ull << 20; }
static bool ntt_mma_pays(int l, uint64_t cols) { return l < 22 && (cols << l) >= 3ull << 20; }
// log2 of the four-step factor n1 that gives the tensor cores the most of a
// 2^l-point transform: both passes where that is possible, else K2 (n1), the
// largest part of an LDE.
static int mma_split(int l) {
    switch (l) {
        case 12: case 13: case 14: case 15: case 16: case 17: return 8;
        case 18: case 19: case 20: case 21: case 22: return 10;
        default: return (l + 1) / 2;
    }
}

size_t ntt_scratch_words(int logn, uint64_t cols) { return logn <= 11 ? 0 : (size_t)cols << logn; }

cudaError_t launch_ntt(const LdePlan& pl, int inverse, uint64_t* data, uint64_t ld, uint64_t cols,
                       uint64_t* scratch, cudaStream_t st, uint64_t* status) {
    const int l = pl.logn;
    const uint64_t* tw12 = pl.tw12_f;  // the inverse negates the sub-DFT input indices instead
    const uint64_t scale = (inverse && l > 0) ? GL_P - ((GL_P - 1) >> l) : 1;  // n^-1 = p - (p-1)/n
    if (cols == 0 || l == 0) return cudaSuccess;  // size-1 transform is the identity
    NvtxRange range(inverse ? "tvmc inverse NTT" : "tvmc forward NTT");
    if (l <= 11) {
        const int lT = choose_lT(l, 11);
        const int T = 1 << lT;
        const size_t smem = words_bytes((1u << l) + spad_words(1 << l, lT));
        return dispatch_ls(l, [&]<int LS>() -> cudaError_t {
            auto kern = inverse ? k_ntt_small<LS, true> : k_ntt_small<LS, false>;
            cudaError_t e = set_smem((const void*)kern, smem);
            if (e != cudaSuccess) return e;
            count_launch();
            kern<<<(unsigned)((cols + T - 1) / T), NTT_THREADS, smem, st>>>(data, ld, cols, lT, tw12, scale);
            return cudaGetLastError();
        });
    }
    const bool mma = ntt_mma_pays(l, cols);
    const int l1 = mma ? mma_split(l) : (l + 1) / 2, l2 = l - l1;
    const uint64_t n = 1ull << l;
    const uint64_t scale_mont = scale == 1 ? 0 : (uint64_t)(((unsigned __int128)scale << 64) % GL_P);
    const uint64_t* wlo = inverse ? pl.wn_i_lo : pl.wn_f_lo;
    const uint64_t* whi = inverse ? pl.wn_i_hi : pl.wn_f_hi;
    const int tile = tuning_ntt_tile_log();
    const int lTa = fit_lT(choose_lT(l2, tile), l2, 1), lTb = fit_lT(choose_lT(l1, tile), l1, 1);
    const size_t smem_a = words_bytes((1u << l2) + spad_words(1 << l2, lTa));
    const size_t smem_b = words_bytes((1u << l1) + spad_words(1 << l1, lTb));
    for (uint64_t c0 = 0; c0 < cols; c0 += 65535) {
        const unsigned nc = (unsigned)((cols - c0) < 65535 ? (cols - c0) : 65535);
        cudaError_t e = mma && lde_mma_size(l2)
                            ? launch_pass_a_mma(l2, pl, inverse, data + c0 * ld, ld, scratch, n, nc, l1, st, status)
                            : dispatch_ls(l2, [&]<int L2>() -> cudaError_t {
            auto kern = inverse ? k_pass_a<L2, true> : k_pass_a<L2, false>;
            cudaError_t e2 = set_smem((const void*)kern, smem_a);
            if (e2 != cudaSuccess) return e2;
            count_launch();
            kern<<<dim3((1u << l1) >> lTa, nc), NTT_THREADS, smem_a, st>>>(data + c0 * ld, ld, scratch, n, l1, lTa,
                                                                          tw12, wlo, whi);
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
        e = mma && lde_mma_size(l1)
                ? launch_pass_b_mma(l1, pl, inverse, scratch, data + c0 * ld, ld, nc, l2, 0, scale_mont, st, status)
                : dispatch_ls(l1, [&]<int L1>() -> cudaError_t {
            auto kern = inverse ? k_pass_b<L1, true> : k_pass_b<L1, false>;
            cudaError_t e2 = set_smem((const void*)kern, smem_b);
            if (e2 != cudaSuccess) return e2;
            count_launch();
            kern<<<dim3((1u << l2) >> lTb, nc), NTT_THREADS, smem_b, st>>>(scratch, n, data + c0 * ld, ld, l2, lTb,
                                                                          tw12, scale);
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

size_t lde_scratch_words(int logn, int log_exp, uint64_t cols) {
    if (logn <= 11) return 0;
    return (size_t)cols * ((size_t)1 << logn) * (1 + ((size_t)1 << log_exp));
}

cudaError_t launch_lde(const LdePlan& pl, const uint64_t* trace, uint64_t tld, uint64_t* out, uint64_t old,
                       uint64_t cols, uint64_t* scratch, cudaStream_t st, uint64_t* status, const uint64_t* add,
                       int rm) {
    const int l = pl.logn, le = pl.log_exp;
    const int hi_len = l > 12 ? (1 << (l - 12)) : 1;
    if (cols == 0) return cudaSuccess;
    NvtxRange range("tvmc LDE");
    if (l <= 11) {
        if (l == 0) {
            const uint64_t total = cols << le;
            count_launch();
            k_lde_one<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(trace, tld, out, old, total, le, add, rm);
            return cudaGetLastError();
        }
        return launch_lde_small(pl, trace, tld, out, old, cols, add, rm, st);
    }
    // four-step split N = n1 * n2 (K2 runs the n1-point transforms, K1 and K3
    // the n2-point ones): the tensor cores' (mma_split) or the balanced one, unless
    // the tuning knob "lde_split_l1" picks another, with both factors at least 2^6 so
    // that a tile of the register networks is never short of sequences (mma_split
    // goes down to n2 = 2^4, where n1 = 2^8 fills the tile)
    const bool mma = tuning_lde_mid_variant() == 3 && lde_mma_pays(l, cols);
    int l1 = mma ? mma_split(l) : (l + 1) / 2;
    if (const int ks = tuning_lde_split_l1(); ks >= 6 && ks <= 12 && l - ks >= 6 && l - ks <= 12) l1 = ks;
    // K3 holds one sequence of every coset per tile: with a large expansion a
    // smaller n2 keeps that tile within shared memory (2^22 rows x 16)
    while (l1 < 12 && ((size_t)(1u << (l - l1)) + spad_words(1 << (l - l1), le)) * 8 > 227 * 1024) l1++;
    const int l2 = l - l1;
    const int tile = tuning_ntt_tile_log();
    const uint64_t N = 1ull << l;
    // passes of 2^8 and 2^10 points run on the tensor cores (lde_mma.cu); K2 for
    // expansions whose per-coset tables fit
    const bool mma_ab = mma && lde_mma_size(l2), mma_mid = mma && lde_mma_size(l1) && le <= lde_mma_max_le(l1);
    const int lT1 = std::min(fit_lT(choose_lT(l2, tile), l2, 1), l1);
    const size_t smem1 = words_bytes((1u << l2) + spad_words(1 << l2, lT1));
    const int lT2 = std::min(fit_lT(choose_lT(l1, tile), l1, 2), l2);
    const size_t smem2 = words_bytes((size_t)(1u << l1) + 2 * spad_words(1 << l1, lT2));
    const int lT3 = std::min(fit_lT(clampi(tile - l2 - le, 0, l2 <= 5 ? 8 - le : 1), l2, 1, le), l1);
    const size_t smem3 = words_bytes((1u << l2) + spad_words(1 << l2, lT3 + le));
    uint64_t* Y = scratch;
    for (uint64_t c0 = 0; c0 < cols; c0 += 65535) {
        const unsigned nc = (unsigned)((cols - c0) < 65535 ? (cols - c0) : 65535);
        uint64_t* Z = scratch + (size_t)nc * N;
        const uint64_t* addc = rm ? add + c0 * ((uint64_t)rm << le) : nullptr;
        cudaError_t e = mma_ab ? launch_pass_a_mma(l2, pl, true, trace + c0 * tld, tld, Y, N, nc, l1, st, status)
                               : dispatch_ls(l2, [&]<int L2>() -> cudaError_t {
            cudaError_t e2 = set_smem((const void*)k_lde_inv_a<L2>, smem1);
            if (e2 != cudaSuccess) return e2;
            count_launch();
            k_lde_inv_a<L2><<<dim3((1u << l1) >> lT1, nc), NTT_THREADS, smem1, st>>>(
                trace + c0 * tld, tld, Y, N, l1, lT1, pl.tw12_f, pl.wn_i_lo, pl.wn_i_hi);
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
        e = mma_mid ? launch_lde_mid_mma(l1, pl, Y, N, Z, nc, l2, hi_len, addc, rm, st, status)
                    : dispatch_ls(l1, [&]<int L1>() -> cudaError_t {
            if constexpr (Plan<L1>::NR == 2 && Plan<L1>::b1 == Plan<L1>::b2) {
                constexpr int lTr = 7 - Plan<L1>::b2;
                if (tuning_lde_mid_variant() != 1) {
                    constexpr size_t R2 = (size_t)1 << Plan<L1>::b2;
                    const size_t sm2 = words_bytes(R2 * (R2 + 1) + spad_words(1 << L1, lTr) +
                                                   ((size_t)1 << (lTr + L1)) + ((size_t)1 << lTr) * (R2 + 1));
                    auto kern = rm ? k_lde_mid_sym2<L1, 2, true>
                                   : (tuning_lde_mid_ctas() == 3 ? k_lde_mid_sym2<L1, 3, false>
                                                                 : k_lde_mid_sym2<L1, 2, false>);
                    cudaError_t e2 = set_smem((const void*)kern, sm2);
                    if (e2 != cudaSuccess) return e2;
                    count_launch();
                    kern<<<dim3((1u << l2) >> lTr, nc), 128, sm2, st>>>(
                        Y, N, Z, l2, le, pl.tw12_f, pl.wn_f_lo, pl.wn_f_hi, pl.sc_lo, pl.sc_hi, hi_len, addc, rm);
                    return cudaGetLastError();
                }
                const size_t smr = words_bytes((size_t)(1u << L1) + spad_words(1 << L1, lTr));
                // register budget: 2 resident CTAs (no spills) or 3 (a few spills); tuning knob
                // (the randomized variant runs at 2 CTAs per SM)
                auto kern = rm ? k_lde_mid_sym<L1, 2, true>
                               : (tuning_lde_mid_ctas() == 3 ? k_lde_mid_sym<L1, 3, false> : k_lde_mid_sym<L1, 2, false>);
                cudaError_t e2 = set_smem((const void*)kern, smr);
                if (e2 != cudaSuccess) return e2;
                count_launch();
                kern<<<dim3((1u << l2) >> lTr, nc), 128, smr, st>>>(
                    Y, N, Z, l2, le, pl.tw12_f, pl.wn_f_lo, pl.wn_f_hi, pl.sc_lo, pl.sc_hi, hi_len,
                    addc, rm);
            } else if constexpr (Plan<L1>::NR == 2) {
                constexpr int lTr = 7 - Plan<L1>::b2;
                const size_t smr = words_bytes((size_t)(1u << L1) + spad_words(1 << L1, lTr));
                auto kern = rm ? k_lde_mid_reg<L1, true> : k_lde_mid_reg<L1, false>;
                cudaError_t e2 = set_smem((const void*)kern, smr);
                if (e2 != cudaSuccess) return e2;
                count_launch();
                kern<<<dim3((1u << l2) >> lTr, nc), 128, smr, st>>>(
                    Y, N, Z, l2, le, pl.tw12_f, pl.wn_f_lo, pl.wn_f_hi, pl.sc_lo, pl.sc_hi, hi_len,
                    addc, rm);
            } else {
                auto kern = rm ? k_lde_mid<L1, true> : k_lde_mid<L1, false>;
                cudaError_t e2 = set_smem((const void*)kern, smem2);
                if (e2 != cudaSuccess) return e2;
                count_launch();
                kern<<<dim3((1u << l2) >> lT2, nc), NTT_THREADS, smem2, st>>>(
                    Y, N, Z, l2, lT2, le, pl.tw12_f, pl.wn_f_lo, pl.wn_f_hi, pl.sc_lo, pl.sc_hi, hi_len,
                    addc, rm);
            }
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
        e = mma_ab ? launch_pass_b_mma(l2, pl, false, Z, out + c0 * old, old, nc, l1, le, 0, st, status)
                   : dispatch_ls(l2, [&]<int L2>() -> cudaError_t {
            cudaError_t e2 = set_smem((const void*)k_lde_fwd_b<L2>, smem3);
            if (e2 != cudaSuccess) return e2;
            count_launch();
            k_lde_fwd_b<L2><<<dim3((1u << l1) >> lT3, nc), NTT_THREADS, smem3, st>>>(Z, out + c0 * old, old, l1,
                                                                                   lT3, le, pl.tw12_f);
            return cudaGetLastError();
        });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ------------------------------------------------------------ coset scale

// 16 consecutive coefficients per thread: one power, then running products.
__global__ void k_coset_scale(const uint64_t* __restrict__ in, uint64_t ild, uint64_t n, uint64_t* __restrict__ out,
                              uint64_t L, uint64_t cols, uint64_t o) {
    const uint64_t per_col = (L + 15) / 16;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < cols * per_col;
         g += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = g / per_col, i0 = (g - c * per_col) * 16;
        uint64_t w = gl_canon(gl_pow(o, i0));
        for (uint64_t i = i0; i < i0 + 16 && i < L; i++) {
            out[c * L + i] = i < n ? gl_mul_c(gl_canon(in[c * ild + i]), w) : 0;
            w = gl_mul_c(w, o);
        }
    }
}

cudaError_t launch_coset_scale(const uint64_t* in, uint64_t ild, uint64_t n, uint64_t* out, uint64_t L, uint64_t cols,
                               uint64_t o, cudaStream_t st) {
    const uint64_t work = cols * ((L + 15) / 16);
    if (work == 0) return cudaSuccess;
    const uint64_t blocks = (work + 255) / 256;
    count_launch();
    k_coset_scale<<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, st>>>(in, ild, n, out, L, cols, o % GL_P);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- transpose

__global__ void k_transpose(const uint64_t* __restrict__ in, uint64_t ild, uint64_t* __restrict__ out,
                            uint64_t old, uint64_t R, uint64_t C) {
    // in: R x C with row stride ild; out: C x R with row stride old.
    __shared__ uint64_t tile[32][33];
    const uint64_t r0 = (uint64_t)blockIdx.y * 32, c0 = (uint64_t)blockIdx.x * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const uint64_t r = r0 + k, c = c0 + threadIdx.x;
        if (r < R && c < C) tile[k][threadIdx.x] = in[r * ild + c];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const uint64_t c = c0 + k, r = r0 + threadIdx.x;
        if (r < R && c < C) out[c * old + r] = tile[threadIdx.x][k];
    }
}

cudaError_t launch_transpose(const uint64_t* in, uint64_t rld, uint64_t* out, uint64_t cld, uint64_t rows,
                             uint64_t cols, cudaStream_t st) {
    if (rows == 0 || cols == 0) return cudaSuccess;
    if (rld == cols && cld == rows && tuning_transpose_tma()) {
        const cudaError_t e = launch_transpose_tma(in, out, rows, cols, st);
        if (e != cudaErrorNotSupported) return e;  // odd sizes fall through to the tile kernel
    }
    // grid.y (row tiles) is limited to 65535: tall tables go in bands of rows
    constexpr uint64_t BAND = 65535ull * 32;
    for (uint64_t r0 = 0; r0 < rows; r0 += BAND) {
        const uint64_t nr = rows - r0 < BAND ? rows - r0 : BAND;
        const dim3 g((unsigned)((cols + 31) / 32), (unsigned)((nr + 31) / 32));
        count_launch();
        k_transpose<<<g, dim3(32, 8), 0, st>>>(in + r0 * rld, rld, out + r0, cld, nr, cols);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_transpose_cm_to_rm(const uint64_t* in, uint64_t cld, uint64_t* out, uint64_t rld,
                                      uint64_t rows, uint64_t cols, cudaStream_t st) {
    if (rows == 0 || cols == 0) return cudaSuccess;
    const dim3 g((unsigned)((rows + 31) / 32), (unsigned)((cols + 31) / 32));
    count_launch();
    k_transpose<<<g, dim3(32, 8), 0, st>>>(in, cld, out, rld, cols, rows);
    return cudaGetLastError();
}

}  // namespace tvmc
