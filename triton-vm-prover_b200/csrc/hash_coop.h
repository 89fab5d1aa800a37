// Launchers of the sixteen-lanes-per-state Tip5 kernels (hash_coop.cu).
#pragma once
#include "internal.cuh"

namespace tvmc {

// Leaf digests as launch_hash_rows, without the tree above them.
cudaError_t launch_hash_rows_coop(const uint64_t* table, uint64_t rstride, uint64_t cstride, uint64_t rows,
                                  uint32_t width, uint64_t* digests, uint64_t* tree, int layout, cudaStream_t st);
// Leaves of several tables; block0 counts CTAs (coop_blocks per table).
cudaError_t launch_hash_jobs_coop(const HashJobs& jobs, uint32_t blocks, cudaStream_t st);
uint64_t coop_blocks(uint64_t rows);
// `levels` <= COOP_TREE_LEVELS levels above the m nodes [m, 2m) in place.
constexpr int COOP_TREE_LEVELS = 7;
cudaError_t launch_merkle_coop(uint64_t* tree, uint64_t n, uint64_t m, int layout, int levels, cudaStream_t st);
// Up to COOP_TREE_LEVELS levels of each of several heap trees; block0 counts CTAs
// (coop_tree_blocks per tree).
cudaError_t launch_merkle_levels_coop(const LevelJobs& jobs, uint32_t blocks, cudaStream_t st);
constexpr uint64_t coop_tree_blocks(uint64_t m) { return (m + (1 << COOP_TREE_LEVELS) - 1) >> COOP_TREE_LEVELS; }
cudaError_t launch_hash_pairs_coop(const uint64_t* left, const uint64_t* right, uint64_t* out, uint64_t count,
                                   cudaStream_t st);
cudaError_t launch_tip5_permutations_coop(uint64_t* states, uint64_t count, cudaStream_t st);

}  // namespace tvmc
