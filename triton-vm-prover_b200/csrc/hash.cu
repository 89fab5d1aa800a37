// Dispatch of the Tip5 row hashing and Merkle tree kernels (sm_100a), and the
// small kernels around them.
//
// Two forms of the permutation carry the path: the tensor-core form, 128 states
// per MMA with two threads each (hash_mma.cu), for throughput, and the
// sixteen-lanes-per-state form (hash_coop.cu), for the latency of few states.
//
// Merkle: parent = hash_pair(left, right) (src/merkle/merkle_tree.cpp:41-61).
// Wide levels take one launch each, the narrow ones COOP_TREE_LEVELS per launch.
#include "hash_coop.h"
#include "hash_mma.h"
#include "internal.cuh"
#include "tip5.cuh"

namespace tvmc {

// Up to this many rows (of all tables of a launch) the sixteen-lane form is
// faster.  379 columns: its time grows from 69 us (up to 1024 rows) by 23 us per
// 1024 rows, while one tile per SM of the tensor-core form takes 314 us however
// many rows it holds; they would meet at about 11600.  At 10240 rows, us
// (sixteen-lane | tensor-core): 9 columns 13.1 | 16.6, 40 41 | 47, 264 199 | 224,
// 379 277 | 314.
constexpr uint64_t COOP_MAX_ROWS = 10240;
// Tree levels with at least this many parents go to the tensor-core form: one
// level takes it 18-20 us up to 16384 parents; the sixteen-lane form takes 12 us
// at 1024 parents, 17 at 4096 and 35 at 16384, and does the levels below in the
// same launch.
constexpr uint64_t MMA_MIN_PARENTS = 8192;

// Leaf i = the in_words words at leaves[in_words*i], zero-padded to a digest:
// in_words = 5 copies digests, 3 turns an XFieldElement into the digest
// (c0, c1, c2, 0, 0), as the reference's FRI trees do (src/fri/fri.cpp:25-43).
__global__ void k_copy_leaves(const uint64_t* __restrict__ leaves, uint64_t* __restrict__ tree, uint64_t n,
                              int layout, int in_words) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t* dst = tree + 5 * node_slot(n + i, n, layout);
#pragma unroll
    for (int k = 0; k < 5; k++) dst[k] = k < in_words ? gl_canon(leaves[(uint64_t)in_words * i + k]) : 0;
}

// Rounds [r0, r0 + nr) on each state; with `trace`, the state after each round
// at trace[(i*nr + k)*16 + .].
__global__ void __launch_bounds__(128) k_tip5_rounds(uint64_t* __restrict__ states, uint64_t count, int r0, int nr,
                                                     uint64_t* __restrict__ trace) {
    __shared__ uint32_t sbox[T5_SBOX_WORDS];
    t5_sbox_init(sbox);
    __syncthreads();
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    uint64_t s[T5_STATE];
#pragma unroll
    for (int k = 0; k < T5_STATE; k++) s[k] = states[16 * i + k];
    for (int k = 0; k < nr; k++) {
        t5_round(s, sbox + (threadIdx.x & 31), r0 + k);
        if (trace) {
#pragma unroll
            for (int j = 0; j < T5_STATE; j++) trace[(i * nr + k) * 16 + j] = gl_canon(s[j]);
        }
    }
#pragma unroll
    for (int k = 0; k < T5_STATE; k++) states[16 * i + k] = gl_canon(s[k]);
}

__global__ void k_gather_auth(const uint64_t* __restrict__ tree, uint64_t n, int layout, int height,
                              const uint64_t* __restrict__ idx, uint64_t count, uint64_t* __restrict__ out) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count * (uint64_t)height) return;
    uint64_t q = t / height;
    int k = (int)(t - q * height);
    uint64_t node = ((n + idx[q]) >> k) ^ 1;
    const uint64_t* src = tree + 5 * node_slot(node, n, layout);
#pragma unroll
    for (int i = 0; i < 5; i++) out[5 * t + i] = src[i];
}

__global__ void k_gather_nodes(const uint64_t* __restrict__ tree, uint64_t n, int layout,
                               const uint64_t* __restrict__ hidx, uint64_t count, uint64_t* __restrict__ out) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const uint64_t* src = tree + 5 * node_slot(hidx[t], n, layout);
#pragma unroll
    for (int i = 0; i < 5; i++) out[5 * t + i] = src[i];
}

__global__ void k_gather_rows(const uint64_t* __restrict__ tab, uint64_t ld, uint32_t width,
                              const uint64_t* __restrict__ rows, uint64_t count, uint64_t* __restrict__ out) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count * (uint64_t)width) return;
    uint64_t q = t / width;
    uint64_t c = t - q * width;
    out[t] = tab[c * ld + rows[q]];
}

static inline int ilog2u(uint64_t x) { return 63 - __builtin_clzll(x); }

static inline unsigned grid_for(uint64_t work, unsigned threads) {
    return (unsigned)((work + threads - 1) / threads);
}

// The m nodes of one level (heap indices [m, 2m)) of a tree with n leaves are
// in place: build every level above.
static cudaError_t launch_tree_above(uint64_t* tree, uint64_t n, uint64_t m, int layout, cudaStream_t st,
                                     uint64_t* status) {
    while (m > 1) {
        int levels = 1;
        cudaError_t e;
        if ((m >> 1) >= MMA_MIN_PARENTS) {
            e = launch_merkle_level_mma(tree, n, m, layout, st, status);
        } else {
            levels = ilog2u(m) < COOP_TREE_LEVELS ? ilog2u(m) : COOP_TREE_LEVELS;
            e = launch_merkle_coop(tree, n, m, layout, levels, st);
        }
        if (e != cudaSuccess) return e;
        m >>= levels;
    }
    return cudaSuccess;
}

cudaError_t launch_hash_rows(const uint64_t* table, uint64_t rstride, uint64_t cstride, uint64_t rows,
                             uint32_t width, uint64_t* digests, uint64_t* tree, int layout,
                             cudaStream_t st, uint64_t* status) {
    if (rows == 0) return cudaSuccess;
    NvtxRange range("tvmc row hash + Merkle tree");
    const cudaError_t e =
        rows <= COOP_MAX_ROWS ? launch_hash_rows_coop(table, rstride, cstride, rows, width, digests, tree, layout, st)
                              : launch_hash_rows_mma(table, rstride, cstride, rows, width, digests, tree, layout, st,
                                                     status);
    return e != cudaSuccess || !tree ? e : launch_tree_above(tree, rows, rows, layout, st, status);
}

// Every level above the leaves of each of count heap trees, all trees in each
// launch, by the rule of one tree (launch_tree_above) on the parents of all.  With
// launches of its own for each tree's wide levels a batch of 64 tables of 2^10 x 4
// (x4) took 1.93 ms, with these 0.59.
static cudaError_t launch_trees_above(const MultiHashTable* tabs, int count, cudaStream_t st) {
    uint64_t m[HASH_MULTI_MAX];
    for (int k = 0; k < count; k++) m[k] = tabs[k].L;
    for (;;) {
        uint64_t parents = 0;
        for (int k = 0; k < count; k++) parents += m[k] >> 1;
        if (parents == 0) return cudaSuccess;
        const bool mma = parents >= MMA_MIN_PARENTS;
        LevelJobs lj{};
        uint64_t blocks = 0;
        for (int k = 0; k < count; k++) {
            if (m[k] < 2) continue;
            lj.j[lj.count++] = LevelJob{tabs[k].tree, m[k], (uint32_t)blocks};
            blocks += mma ? mma_tiles(m[k] >> 1) : coop_tree_blocks(m[k]);
            m[k] >>= mma ? 1 : (ilog2u(m[k]) < COOP_TREE_LEVELS ? ilog2u(m[k]) : COOP_TREE_LEVELS);
        }
        const cudaError_t e = mma ? launch_merkle_levels_mma(lj, (uint32_t)blocks, st)
                                  : launch_merkle_levels_coop(lj, (uint32_t)blocks, st);
        if (e != cudaSuccess) return e;
    }
}

cudaError_t launch_hash_rows_multi(const MultiHashTable* tabs, int count, cudaStream_t st) {
    NvtxRange range("tvmc multi-table row hash + Merkle trees");
    for (int c0 = 0; c0 < count; c0 += HASH_MULTI_MAX) {
        const int nj = count - c0 < HASH_MULTI_MAX ? count - c0 : HASH_MULTI_MAX;
        uint64_t rows = 0;
        for (int k = 0; k < nj; k++) rows += tabs[c0 + k].L;
        const bool coop = rows <= COOP_MAX_ROWS;
        HashJobs hj{};
        uint64_t blocks = 0;
        for (int k = 0; k < nj; k++) {
            const MultiHashTable& t = tabs[c0 + k];
            hj.j[k] = HashJob{t.lde, t.tree, t.L, t.width, (uint32_t)blocks};
            blocks += coop ? coop_blocks(t.L) : mma_tiles(t.L);
        }
        hj.count = nj;
        if (blocks == 0) continue;
        cudaError_t e = coop ? launch_hash_jobs_coop(hj, (uint32_t)blocks, st)
                             : launch_hash_jobs_mma(hj, (uint32_t)blocks, st);
        if (e == cudaSuccess) e = launch_trees_above(tabs + c0, nj, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_merkle_tree(const uint64_t* leaves, uint64_t* tree, uint64_t n, int layout,
                               cudaStream_t st, uint64_t* status, int leaf_words) {
    count_launch();
    k_copy_leaves<<<grid_for(n, 256), 256, 0, st>>>(leaves, tree, n, layout, leaf_words);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_tree_above(tree, n, n, layout, st, status);
}

cudaError_t launch_hash_pairs(const uint64_t* left, const uint64_t* right, uint64_t* out, uint64_t count,
                              cudaStream_t st, uint64_t* status) {
    if (count == 0) return cudaSuccess;
    return count < MMA_MIN_PARENTS ? launch_hash_pairs_coop(left, right, out, count, st)
                                   : launch_hash_pairs_mma(left, right, out, count, st, status);
}

cudaError_t launch_tip5_permutations(uint64_t* states, uint64_t count, cudaStream_t st, uint64_t* status) {
    if (count == 0) return cudaSuccess;
    return count < MMA_MIN_PARENTS ? launch_tip5_permutations_coop(states, count, st)
                                   : launch_tip5_permutations_mma(states, count, st, status);
}

cudaError_t launch_tip5_rounds(uint64_t* states, uint64_t count, int r0, int nr, uint64_t* trace, cudaStream_t st) {
    if (count == 0 || nr == 0) return cudaSuccess;
    count_launch();
    k_tip5_rounds<<<grid_for(count, 128), 128, 0, st>>>(states, count, r0, nr, trace);
    return cudaGetLastError();
}

cudaError_t launch_gather_auth_paths(const uint64_t* tree, uint64_t n, int layout, const uint64_t* idx,
                                     uint64_t count, uint64_t* out, cudaStream_t st) {
    int height = ilog2u(n);
    if (count == 0 || height == 0) return cudaSuccess;
    count_launch();
    k_gather_auth<<<grid_for(count * height, 256), 256, 0, st>>>(tree, n, layout, height, idx, count, out);
    return cudaGetLastError();
}

cudaError_t launch_gather_nodes(const uint64_t* tree, uint64_t n, int layout, const uint64_t* heap_idx,
                                uint64_t count, uint64_t* out, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    count_launch();
    k_gather_nodes<<<grid_for(count, 256), 256, 0, st>>>(tree, n, layout, heap_idx, count, out);
    return cudaGetLastError();
}

cudaError_t launch_gather_rows(const uint64_t* table, uint64_t ld, uint32_t width, const uint64_t* rows,
                               uint64_t count, uint64_t* out, cudaStream_t st) {
    if (count == 0 || width == 0) return cudaSuccess;
    count_launch();
    k_gather_rows<<<grid_for(count * width, 256), 256, 0, st>>>(table, ld, width, rows, count, out);
    return cudaGetLastError();
}

cudaError_t launch_absorb_stripe(const uint64_t* stripe, uint64_t L, uint32_t ncols, uint64_t* cap, int first,
                                 int last, uint64_t* tree, cudaStream_t st) {
    NvtxRange range("tvmc frugal stripe absorb");
    const cudaError_t e = launch_absorb_stripe_mma(stripe, L, ncols, cap, first, last, tree, st);
    return e != cudaSuccess || !last ? e : launch_tree_above(tree, L, L, LAYOUT_HEAP, st, tree);
}

}  // namespace tvmc
