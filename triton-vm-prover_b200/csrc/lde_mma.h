// Launchers of the tensor-core transform passes (lde_mma.cu): sub-transforms of
// 2^8 and 2^10 points (two rounds of radix 16 or 32).
#pragma once
#include "internal.cuh"

namespace tvmc {

constexpr bool lde_mma_size(int lsub) { return lsub == 8 || lsub == 10; }
// Largest log2 expansion of launch_lde_mid_mma, whose per-coset tables share the SM.
constexpr int lde_mma_max_le(int lsub) { return lsub == 10 ? 2 : 4; }

// Pass A with n2 = 2^lsub, n1 = 2^l1 >= 8 (ntt.cu, k_lde_inv_a and k_pass_a).
cudaError_t launch_pass_a_mma(int lsub, const LdePlan& pl, bool inverse, const uint64_t* in, uint64_t ild, uint64_t* Y,
                              uint64_t yld, uint32_t cols, int l1, cudaStream_t st, uint64_t* status);
// K2 with n1 = 2^lsub, n2 = 2^l2 >= 8; add, rm: launch_lde's randomizer addends of these columns.
cudaError_t launch_lde_mid_mma(int lsub, const LdePlan& pl, const uint64_t* Y, uint64_t yld, uint64_t* Z, uint32_t cols,
                               int l2, int hi_len, const uint64_t* add, int rm, cudaStream_t st, uint64_t* status);
// Pass B over rows of 2^lsub points, 2^l1 >= 8 rows per coset (k_lde_fwd_b; le = 0:
// k_pass_b); an inverse's outputs times scale_mont (Montgomery form).
cudaError_t launch_pass_b_mma(int lsub, const LdePlan& pl, bool inverse, const uint64_t* Z, uint64_t* out, uint64_t old,
                              uint32_t cols, int l1, int le, uint64_t scale_mont, cudaStream_t st,
                              uint64_t* status);
unsigned int lde_mma_timeouts();

}  // namespace tvmc
