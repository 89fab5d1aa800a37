// In-CTA sub-transforms on register networks, shared by the NTT and LDE kernels
// (ntt.cu describes the structure).
#pragma once
#include "field.cuh"
#include "internal.cuh"

namespace tvmc {

constexpr int NTT_THREADS = 256;

// ------------------------------------------------------------ sub-transform

// Shared-memory slot of element k (T = 2^lT interleaved sequences); one row of
// padding per 32 elements keeps every round's line accesses bank-conflict free.
__device__ __forceinline__ int spos(int k, int lT) { return (k + (k >> 5)) << lT; }
// The slot of k = a + (b << BITS) with a < 2^BITS: for BITS = 5 the padding
// term k >> 5 is b itself, so the slot is (a + 33 b) << lT -- an index the
// compiler can split into a per-line base and per-element constants.
template <int BITS>
__device__ __forceinline__ int spos2(int a, int b, int lT) {
    if constexpr (BITS == 5) return (a + 33 * b) << lT;
    else return spos(a + (b << BITS), lT);
}
__host__ __device__ constexpr int spad_words(int n, int lT) { return (n + (n >> 5) + 1) << lT; }

// Round sizes (log2) of a 2^LS transform: one round up to 2^5, two up to 2^10,
// three beyond.  b1 is the last round (contiguous digit).
template <int LS>
struct Plan {
    static constexpr int NR = LS <= 5 ? 1 : (LS <= 10 ? 2 : 3);
    static constexpr int b1 = NR == 1 ? LS : (NR == 2 ? LS - LS / 2 : (LS + 2) / 3);
    static constexpr int b2 = NR == 1 ? 0 : (NR == 2 ? LS / 2 : (LS + 1) / 3);
    static constexpr int b3 = NR == 3 ? LS / 3 : 0;
    static_assert(b1 + b2 + b3 == LS, "round split");
    static_assert(b1 <= 5 && b2 <= 5 && b3 <= 5, "radix <= 32");
};

template <int B>
__device__ __forceinline__ constexpr int brevc(int k) {
    int r = 0;
    for (int i = 0; i < B; i++) r |= ((k >> i) & 1) << (B - 1 - i);
    return r;
}

// The forward 32-point root w_32 = 7^((p-1)/32) is 2^78 (mod p); every root of
// order 2^m <= 32 is its power 2^(78 * 2^(5-m) mod 192).
constexpr int W32_LOG2 = 78;

// Radix-2 DIF network on R = 2^B registers (forward root); X[k] ends in
// v[brev(k)].  Its twiddles w_{2h}^j are roots of order <= 32, applied as
// powers of two (gl_sub_mul_pow2_c): no table, no general multiply.  Every
// inverse transform here runs through the same forward networks on
// index-negated input: DFT_{w^-1}(x)[k] = DFT_w(x')[k] with x'[i] = x[-i mod n].
template <int B>
__device__ __forceinline__ void reg_dft(uint64_t (&v)[1 << B]) {
#pragma unroll
    for (int st = 0; st < B; st++) {
        constexpr int R = 1 << B;
        const int h = R >> (st + 1);
#pragma unroll
        for (int blk = 0; blk < R; blk += 2 * h) {
#pragma unroll
            for (int j = 0; j < h; j++) {
                const uint64_t a = v[blk + j], c = v[blk + j + h];
                v[blk + j] = gl_add_c(a, c);
                v[blk + j + h] = gl_sub_mul_pow2_c(a, c, (W32_LOG2 * j * (16 / h)) % 192);
            }
        }
    }
}

// x times a twiddle from a table: plain (canonical product) or, with MONT, a
// table in Montgomery form (gl_mont_mul: seven fewer instructions).
template <bool MONT>
__device__ __forceinline__ uint64_t tw_mul(uint64_t x, uint64_t w) {
    if constexpr (MONT) return gl_mont_mul(x, w);
    else return gl_mul_c(x, w);
}

// DFT of size 2^LS on T = 2^lT sequences.  load(k, t) returns input element k
// of sequence t (called once per element, by the first round); store(k, t, v)
// receives output X[k] of sequence t (called once, by the last round).  With
// TO_SMEM the last round instead writes X[k] back into s at element slot
// out_pos<LS>(k) (the slots its line read), for a caller's rolled output loop
// after a __syncthreads().  s is a shared buffer of spad_words(2^LS, lT) words
// for the transposes between rounds and tw holds w^e, e < 2^LS.  Callers must
// __syncthreads() before reusing s or before reading, in another thread,
// anything a store wrote to shared memory.  The transform is the forward one
// (tw holds powers of the forward root; callers negate input indices for an
// inverse).
template <int LS, bool TO_SMEM = false, bool MONT = false, class LoadF, class StoreF>
__device__ __forceinline__ void sub_dft(uint64_t* s, int lT, const uint64_t* tw, LoadF&& load, StoreF&& store) {
    using PL = Plan<LS>;
    const int T = 1 << lT;
    if constexpr (PL::NR == 1) {
        constexpr int R = 1 << LS;
        for (int t = threadIdx.x; t < T; t += blockDim.x) {
            uint64_t v[R];
#pragma unroll
            for (int j = 0; j < R; j++) v[j] = load(j, t);
            reg_dft<LS>(v);
#pragma unroll
            for (int k = 0; k < R; k++) {
                if constexpr (TO_SMEM) s[spos(k, lT) + t] = v[brevc<LS>(k)];
                else store(k, t, v[brevc<LS>(k)]);
            }
        }
    } else if constexpr (PL::NR == 2) {
        constexpr int b1 = PL::b1, b2 = PL::b2, R1 = 1 << b1, R2 = 1 << b2;
        // round 1: digit 2 (stride R1) for each (t, d1), twiddle w^(d1*k2)
        for (int id = threadIdx.x; id < (R1 << lT); id += blockDim.x) {
            const int t = id & (T - 1), d1 = id >> lT;
            uint64_t v[R2];
#pragma unroll
            for (int j = 0; j < R2; j++) v[j] = load(d1 + (j << b1), t);
            reg_dft<b2>(v);
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) {
                uint64_t x = v[brevc<b2>(k2)];
                if (k2) x = tw_mul<MONT>(x, tw[d1 * k2]);
                s[spos2<b1>(d1, k2, lT) + t] = x;
            }
        }
        __syncthreads();
        // round 2: digit 1 (contiguous) for each (t, k2) -> X[R2*k1 + k2]
        for (int id = threadIdx.x; id < (R2 << lT); id += blockDim.x) {
            const int t = id & (T - 1), k2 = id >> lT;
            uint64_t v[R1];
#pragma unroll
            for (int d1 = 0; d1 < R1; d1++) v[d1] = s[spos2<b1>(d1, k2, lT) + t];
            reg_dft<b1>(v);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) {
                if constexpr (TO_SMEM) s[spos2<b1>(k1, k2, lT) + t] = v[brevc<b1>(k1)];
                else store((k1 << b2) + k2, t, v[brevc<b1>(k1)]);
            }
        }
    } else {
        constexpr int b1 = PL::b1, b2 = PL::b2, b3 = PL::b3;
        constexpr int R1 = 1 << b1, R2 = 1 << b2, R3 = 1 << b3;
        // round A: digit 3 (stride R1*R2) for each (t, lo = d1 + R1*d2), twiddle w_{R2R3}^(d2*k3)
        for (int id = threadIdx.x; id < ((R1 * R2) << lT); id += blockDim.x) {
            const int t = id & (T - 1), lo = id >> lT;
            uint64_t v[R3];
#pragma unroll
            for (int j = 0; j < R3; j++) v[j] = load(lo + (j << (b1 + b2)), t);
            reg_dft<b3>(v);
#pragma unroll
            for (int k3 = 0; k3 < R3; k3++) {
                uint64_t x = v[brevc<b3>(k3)];
                const int e = ((lo >> b1) * k3) << b1;
                if (e) x = tw_mul<MONT>(x, tw[e]);
                s[spos(lo + (k3 << (b1 + b2)), lT) + t] = x;
            }
        }
        __syncthreads();
        // round B: digit 2 (stride R1) for each (t, d1, k3), twiddle w^(d1*(R3*k2 + k3))
        for (int id = threadIdx.x; id < ((R1 * R3) << lT); id += blockDim.x) {
            const int t = id & (T - 1), rest = id >> lT;
            const int d1 = rest & (R1 - 1), k3 = rest >> b1;
            const int base = d1 + (k3 << (b1 + b2));
            uint64_t v[R2];
#pragma unroll
            for (int j = 0; j < R2; j++) v[j] = s[spos(base + (j << b1), lT) + t];
            reg_dft<b2>(v);
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) {
                uint64_t x = v[brevc<b2>(k2)];
                const int e = d1 * (R3 * k2 + k3);
                if (e) x = tw_mul<MONT>(x, tw[e]);
                s[spos(base + (k2 << b1), lT) + t] = x;
            }
        }
        __syncthreads();
        // round C: digit 1 (contiguous) for each (t, k2, k3) -> X[R2R3*k1 + R3*k2 + k3]
        for (int id = threadIdx.x; id < ((R2 * R3) << lT); id += blockDim.x) {
            const int t = id & (T - 1), rest = id >> lT;
            const int k2 = rest & (R2 - 1), k3 = rest >> b2;
            uint64_t v[R1];
#pragma unroll
            for (int d1 = 0; d1 < R1; d1++) v[d1] = s[spos(d1 + (rest << b1), lT) + t];
            reg_dft<b1>(v);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) {
                if constexpr (TO_SMEM) s[spos(k1 + (rest << b1), lT) + t] = v[brevc<b1>(k1)];
                else store((k1 << (b2 + b3)) + R3 * k2 + k3, t, v[brevc<b1>(k1)]);
            }
        }
    }
}

// Element slot of X[k] after sub_dft<LS, true>.
template <int LS>
__device__ __forceinline__ int out_pos(int k) {
    using PL = Plan<LS>;
    if constexpr (PL::NR == 1) {
        return k;
    } else if constexpr (PL::NR == 2) {
        return (k >> PL::b2) + ((k & ((1 << PL::b2) - 1)) << PL::b1);  // X[R2*k1 + k2] at k1 + R1*k2
    } else {
        const int k1 = k >> (PL::b2 + PL::b3);  // X[M*k1 + R3*k2 + k3] at k1 + R1*(k2 + R2*k3)
        const int k2 = (k >> PL::b3) & ((1 << PL::b2) - 1);
        const int k3 = k & ((1 << PL::b3) - 1);
        return k1 + ((k2 + (k3 << PL::b2)) << PL::b1);
    }
}

__device__ __forceinline__ uint64_t tw2(const uint64_t* __restrict__ lo, const uint64_t* __restrict__ hi,
                                        uint32_t e) {
    return gl_mul(__ldg(lo + (e & 4095)), __ldg(hi + (e >> 12)));
}

// tw[e] = w_{2^LS}^e, e < 2^LS, from the 4096-entry table of w_4096 powers
// (with MONT in Montgomery form, w * 2^64).
template <int LS, bool MONT = false>
__device__ __forceinline__ void load_tw(uint64_t* tw, const uint64_t* __restrict__ tw12) {
    for (int m = threadIdx.x; m < (1 << LS); m += blockDim.x) {
        const uint64_t w = __ldg(tw12 + (m << (12 - LS)));
        tw[m] = MONT ? gl_to_mont(w) : w;
    }
}

// Lets a launch of fn (a kernel without static shared memory) take `bytes` of
// dynamic shared memory.
inline cudaError_t set_smem(const void* fn, size_t bytes) {
    return bytes > 48 * 1024 ? raise_smem_limit(fn) : cudaSuccess;
}

// Calls F.template operator()<L>() for the runtime L in [1, 12].
template <typename F>
cudaError_t dispatch_ls(int l, F&& f) {
    switch (l) {
        case 1: return f.template operator()<1>();
        case 2: return f.template operator()<2>();
        case 3: return f.template operator()<3>();
        case 4: return f.template operator()<4>();
        case 5: return f.template operator()<5>();
        case 6: return f.template operator()<6>();
        case 7: return f.template operator()<7>();
        case 8: return f.template operator()<8>();
        case 9: return f.template operator()<9>();
        case 10: return f.template operator()<10>();
        case 11: return f.template operator()<11>();
        case 12: return f.template operator()<12>();
        default: return cudaErrorInvalidValue;
    }
}

inline size_t words_bytes(size_t w) { return w * 8; }

}  // namespace tvmc
