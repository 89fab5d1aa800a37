// Tip5 permutation with sixteen lanes per state (sm_100a): the low-latency form.
//
// A call with few states (a short table's rows, a tree's upper levels, one
// sponge) is bound by the length of one permutation's dependence chain, not by
// throughput.  Here lane l of a half-warp holds state word l: x^7 and the byte
// lookups of all words run side by side, the words go to the half-warp's
// exchange buffer in shared memory as pairs of exact doubles, and each lane
// forms its own output word of the MDS.  Sums of 16-bit matrix entries times
// 32-bit halves stay below 524757 * 2^32 < 2^52, so they are exact on the FP64
// pipe without centring.  Per state it issues about 2.5 times the instructions
// of the tensor-core form and takes a quarter of its latency: 2.0 us a
// permutation (B200) against 8.4 (9.0 with one thread per state).  The exchange as
// 64-bit words with integer sums measured 0.080 ms against 0.077 at 1024 rows x
// 379 and 0.285 against 0.235 at 8192.
#pragma once
#include <cstdint>
#include "field.cuh"
#include "tip5.cuh"

namespace tvmc {

constexpr int T5C_LANES = 16;  // threads per state

// Shared tables of a CTA: the byte table in eight interleaved copies (one per
// looking-up lane of a warp, so its lookups fall into distinct banks) and the
// round biases 2^52 + (constant's halves), as t5_recombine expects them.
struct T5CoopTables {
    uint32_t sbox[256 * 8];
    double2 bias[T5_ROUNDS * T5_STATE];
};

// A lane's constant part: its row of the MDS matrix, M[(l - c) mod 16].
struct T5Coop {
    double m[T5_STATE];
    const uint32_t* tbl;     // this lane's copy of the byte table
    const double2* bias;     // this lane's biases, stride T5_STATE
    double2* xch;            // the state's exchange buffer, 2 x 16 entries
    int lane;                // word index, 0..15
};

// Every thread of the CTA calls this once; xch: 32 entries per state of the CTA.
__device__ __forceinline__ void t5c_init(T5Coop& c, T5CoopTables& t, double2* xch) {
    for (int i = threadIdx.x; i < 256 * 8; i += blockDim.x) t.sbox[i] = __ldg(&g_t5_sbox.v[i >> 3]);
    for (int i = threadIdx.x; i < T5_ROUNDS * T5_STATE; i += blockDim.x)
        t.bias[i] = make_double2(__ldg(&g_t5_coop_bias.lo[i]), __ldg(&g_t5_coop_bias.hi[i]));
    c.lane = threadIdx.x & (T5C_LANES - 1);
#pragma unroll
    for (int k = 0; k < T5_STATE; k++) c.m[k] = __ldg(&g_t5_mds_row.v[c.lane - k + T5_STATE]);
    c.tbl = t.sbox + ((threadIdx.x >> 2) & 4) + (c.lane & 3);
    c.bias = t.bias + c.lane;
    c.xch = xch + (threadIdx.x / T5C_LANES) * 2 * T5_STATE;
    __syncthreads();
}

__device__ __forceinline__ uint32_t t5c_lookup32(uint32_t m, const uint32_t* tbl) {
    const uint32_t w0 = tbl[__byte_perm(m, 0, 0x4440) << 3];
    const uint32_t w1 = tbl[__byte_perm(m, 0, 0x4441) << 3];
    const uint32_t w2 = tbl[__byte_perm(m, 0, 0x4442) << 3];
    const uint32_t w3 = tbl[__byte_perm(m, 0, 0x4443) << 3];
    return __byte_perm(__byte_perm(w0, w1, 0x0040), __byte_perm(w2, w3, 0x0040), 0x5410);
}

// The permutation of a state held one Montgomery-form word per lane (any
// representative in and out).  Whole warps call it together.
__device__ __forceinline__ uint64_t t5c_permutation(uint64_t x, const T5Coop& c) {
#pragma unroll 1
    for (int rnd = 0; rnd < T5_ROUNDS; rnd++) {
        const double2 b = c.bias[rnd * T5_STATE];
        // every lane takes both forms of the S-box, so that the lookups overlap the
        // products (as a branch of four lanes: 1024 rows x 379 in 88 us against 77)
        const uint64_t z = gl_canon(x);
        const uint32_t z0 = t5c_lookup32((uint32_t)z, c.tbl), z1 = t5c_lookup32((uint32_t)(z >> 32), c.tbl);
        uint64_t y = t5_pow7_m(x);
        y = c.lane < 4 ? ((uint64_t)z1 << 32) | z0 : y;
        double2* xc = c.xch + (rnd & 1) * T5_STATE;  // two buffers: one warp barrier per round
        constexpr double two52 = 4503599627370496.0;
        xc[c.lane] = make_double2(t5_half_biased((uint32_t)y) - two52, t5_half_biased((uint32_t)(y >> 32)) - two52);
        __syncwarp();
        double l0 = b.x, h0 = b.y, l1 = 0.0, h1 = 0.0;
#pragma unroll
        for (int k = 0; k < T5_STATE; k += 2) {
            const double2 u = xc[k], v = xc[k + 1];
            l0 = fma(c.m[k], u.x, l0);
            h0 = fma(c.m[k], u.y, h0);
            l1 = fma(c.m[k + 1], v.x, l1);
            h1 = fma(c.m[k + 1], v.y, h1);
        }
        x = t5_recombine(l0 + l1, h0 + h1);
    }
    return x;
}

// Writes after a permutation's last round read the first buffer again only after
// the barrier of the round between (five rounds: rounds 0, 2 and 4 use buffer 0),
// so a following permutation needs a barrier of its own before its first write.
__device__ __forceinline__ void t5c_sync() { __syncwarp(); }

// hash_pair of two plain digests: lane l < 5 passes left[l], 5 <= l < 10
// right[l - 5] (other lanes anything); lanes 0..4 return the canonical digest.
__device__ __forceinline__ uint64_t t5c_hash_pair(uint64_t w, const T5Coop& c) {
    t5c_sync();
    return gl_from_mont(t5c_permutation(c.lane < T5_RATE ? gl_to_mont(w) : T5_MONT_ONE, c));
}

}  // namespace tvmc
