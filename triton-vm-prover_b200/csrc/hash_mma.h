// Launchers of the tensor-core Tip5 kernels (hash_mma.cu).
#pragma once
#include "internal.cuh"

namespace tvmc {

// Leaf digests as launch_hash_rows, without the tree above them.
cudaError_t launch_hash_rows_mma(const uint64_t* table, uint64_t rstride, uint64_t cstride, uint64_t rows,
                                 uint32_t width, uint64_t* digests, uint64_t* tree, int layout, cudaStream_t st,
                                 uint64_t* status);
// Leaves of several tables; block0 counts tiles of 128 rows, `tiles` in all.
cudaError_t launch_hash_jobs_mma(const HashJobs& jobs, uint32_t tiles, cudaStream_t st);
// One frugal stripe; `last` writes the leaves, without the tree above them.
cudaError_t launch_absorb_stripe_mma(const uint64_t* stripe, uint64_t L, uint32_t ncols, uint64_t* cap, int first,
                                     int last, uint64_t* tree, cudaStream_t st);
// The level of m/2 parents above the m nodes [m, 2m) in place.
cudaError_t launch_merkle_level_mma(uint64_t* tree, uint64_t n, uint64_t m, int layout, cudaStream_t st,
                                    uint64_t* status);
// The same for several heap trees; block0 counts tiles of 128 parents, `tiles` in all.
cudaError_t launch_merkle_levels_mma(const LevelJobs& jobs, uint32_t tiles, cudaStream_t st);
uint64_t mma_tiles(uint64_t rows);
cudaError_t launch_hash_pairs_mma(const uint64_t* left, const uint64_t* right, uint64_t* out, uint64_t count,
                                  cudaStream_t st, uint64_t* status);
cudaError_t launch_tip5_permutations_mma(uint64_t* states, uint64_t count, cudaStream_t st, uint64_t* status);
// Waits for an MMA that ran out so far (all kernels of this device).
unsigned int mma_timeouts();

}  // namespace tvmc
