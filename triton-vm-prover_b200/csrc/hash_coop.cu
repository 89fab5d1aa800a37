// Tip5 kernels for few states: sixteen lanes per state (tip5_coop.cuh).
//
// The rows of a short table, the upper levels of a tree, openings and sponges
// have too few states to fill the GPU, so their time is the length of the
// permutation chain: these kernels trade about 2.5 times the instructions per
// permutation for a quarter of its latency (the dispatch rules stand in hash.cu).
#include "hash_coop.h"
#include "internal.cuh"
#include "tip5_coop.cuh"

namespace tvmc {

constexpr int COOP_THREADS = 128;                            // 8 states: many small CTAs spread over the SMs
constexpr int COOP_STATES = COOP_THREADS / T5C_LANES;
constexpr int COOP_TREE_THREADS = 512;                       // 32 parents per pass
constexpr int COOP_TREE_STATES = COOP_TREE_THREADS / T5C_LANES;
constexpr int COOP_TREE_NODES = 1 << COOP_TREE_LEVELS;       // nodes per CTA of k_merkle_coop

namespace {

// hash_varlen of one row (element i at p[i * cs]); returns the plain digest in
// lanes 0..4.  The lane's word of the next chunk is loaded one permutation ahead.
__device__ __forceinline__ uint64_t hash_row(const uint64_t* __restrict__ p, uint64_t cs, uint32_t width, bool live,
                                             const T5Coop& c) {
    const bool rate = c.lane < T5_RATE;
    auto word = [&](uint32_t k) -> uint64_t {  // Montgomery form of this lane's word of chunk k
        const uint32_t i = k * T5_RATE + c.lane;
        return i < width ? (live ? gl_to_mont(__ldg(p + (uint64_t)i * cs)) : 0) : (i == width ? T5_MONT_ONE : 0);
    };
    uint64_t x = 0, nx = rate ? word(0) : 0;
    const uint32_t perms = width / T5_RATE + 1;
    for (uint32_t k = 0; k < perms; k++) {
        if (rate) {
            x = nx;
            if (k + 1 < perms) nx = word(k + 1);
        }
        t5c_sync();
        x = t5c_permutation(x, c);
    }
    return gl_from_mont(x);
}

}  // namespace

__global__ void __launch_bounds__(COOP_THREADS) k_hash_rows_coop(const uint64_t* __restrict__ tab, uint64_t rstride,
                                                                 uint64_t cstride, uint64_t rows, uint32_t width,
                                                                 uint64_t* __restrict__ digests,
                                                                 uint64_t* __restrict__ tree, int layout) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_STATES * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    const uint64_t row = (uint64_t)blockIdx.x * COOP_STATES + threadIdx.x / T5C_LANES;
    const bool live = row < rows;
    const uint64_t d = hash_row(tab + (live ? row : 0) * rstride, cstride, width, live, c);
    if (live && c.lane < 5) (tree ? tree + 5 * node_slot(rows + row, rows, layout) : digests + 5 * row)[c.lane] = d;
}

// Up to HASH_MULTI_MAX tables; CTA b belongs to job j with block0[j] <= b < block0[j + 1].
__global__ void __launch_bounds__(COOP_THREADS) k_hash_rows_multi_coop(const __grid_constant__ HashJobs jobs) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_STATES * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    int j = 0;
    for (int k = 1; k < jobs.count; k++)
        if (jobs.j[k].block0 <= blockIdx.x) j = k;
    const uint64_t L = jobs.j[j].L;
    const uint64_t row = (uint64_t)(blockIdx.x - jobs.j[j].block0) * COOP_STATES + threadIdx.x / T5C_LANES;
    const bool live = row < L;
    const uint64_t d = hash_row(jobs.j[j].lde + (live ? row : 0), L, jobs.j[j].width, live, c);
    if (live && c.lane < 5) jobs.j[j].tree[5 * (L + row) + c.lane] = d;
}

namespace {

// Builds the levels above the m nodes in place (heap nodes [m, 2m)) that hang
// under this CTA's chunk of up to COOP_TREE_NODES of them, down to `levels`.
__device__ __forceinline__ void subtree(uint64_t* __restrict__ tree, uint64_t n, uint64_t m, int layout, int levels,
                                        uint64_t chunk, uint64_t* sd, const T5Coop& c) {
    uint32_t cnt = m < COOP_TREE_NODES ? (uint32_t)m : COOP_TREE_NODES;
    uint64_t first = m + chunk * COOP_TREE_NODES;  // heap index of the chunk's first node
    uint64_t *in = sd, *out = sd + 5 * COOP_TREE_NODES;
    for (uint32_t i = threadIdx.x; i < 5 * cnt; i += COOP_TREE_THREADS)
        in[i] = tree[5 * node_slot(first + i / 5, n, layout) + i % 5];
    __syncthreads();
    for (int lv = 0; lv < levels; lv++) {
        cnt >>= 1;
        first >>= 1;
        for (uint32_t b = 0; b < cnt; b += COOP_TREE_STATES) {
            const uint32_t st = b + threadIdx.x / T5C_LANES;
            if ((st & ~1u) >= cnt) continue;  // whole warps: states st and st ^ 1
            const uint32_t s0 = st < cnt ? st : cnt - 1;
            const uint64_t d = t5c_hash_pair(c.lane < T5_RATE ? in[10 * s0 + c.lane] : 0, c);
            if (st < cnt && c.lane < 5) {
                out[5 * st + c.lane] = d;
                tree[5 * node_slot(first + st, n, layout) + c.lane] = d;
            }
        }
        __syncthreads();
        uint64_t* t = in;
        in = out;
        out = t;
    }
}

}  // namespace

__global__ void __launch_bounds__(COOP_TREE_THREADS) k_merkle_coop(uint64_t* __restrict__ tree, uint64_t n, uint64_t m,
                                                                   int layout, int levels) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_TREE_STATES * 2 * T5_STATE];
    __shared__ uint64_t sd[5 * (COOP_TREE_NODES + COOP_TREE_NODES / 2)];
    T5Coop c;
    t5c_init(c, tables, xch);
    subtree(tree, n, m, layout, levels, blockIdx.x, sd, c);
}

// Several heap trees; CTA b belongs to job j with block0[j] <= b < block0[j + 1].
__global__ void __launch_bounds__(COOP_TREE_THREADS) k_merkle_levels_coop(const __grid_constant__ LevelJobs jobs) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_TREE_STATES * 2 * T5_STATE];
    __shared__ uint64_t sd[5 * (COOP_TREE_NODES + COOP_TREE_NODES / 2)];
    T5Coop c;
    t5c_init(c, tables, xch);
    int j = 0;
    for (int k = 1; k < jobs.count; k++)
        if (jobs.j[k].block0 <= blockIdx.x) j = k;
    const uint64_t m = jobs.j[j].m;
    const int lg = 63 - __clzll((long long)m);
    subtree(jobs.j[j].tree, m, m, LAYOUT_HEAP, lg < COOP_TREE_LEVELS ? lg : COOP_TREE_LEVELS,
            blockIdx.x - jobs.j[j].block0, sd, c);
}

__global__ void __launch_bounds__(COOP_THREADS) k_hash_pairs_coop(const uint64_t* __restrict__ left,
                                                                  const uint64_t* __restrict__ right,
                                                                  uint64_t* __restrict__ out, uint64_t count) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_STATES * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    const uint64_t i = (uint64_t)blockIdx.x * COOP_STATES + threadIdx.x / T5C_LANES, k = i < count ? i : count - 1;
    const uint64_t w = c.lane < 5 ? left[5 * k + c.lane] : (c.lane < T5_RATE ? right[5 * k + c.lane - 5] : 0);
    const uint64_t d = t5c_hash_pair(w, c);
    if (i < count && c.lane < 5) out[5 * i + c.lane] = d;
}

__global__ void __launch_bounds__(COOP_THREADS) k_tip5_perm_coop(uint64_t* __restrict__ states, uint64_t count) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_STATES * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    const uint64_t i = (uint64_t)blockIdx.x * COOP_STATES + threadIdx.x / T5C_LANES;
    const bool live = i < count;
    uint64_t x = live ? gl_to_mont(states[T5_STATE * i + c.lane]) : 0;
    x = gl_from_mont(t5c_permutation(x, c));
    if (live) states[T5_STATE * i + c.lane] = x;
}

// Root implied by leaf q and its authentication path (MerkleTree::verify,
// src/merkle/merkle_tree.cpp:343-364): paths[(q*len + k)*5 + .] is the sibling
// at height k; leaf index bit k says which side the running digest is on.  The
// chain of a path favours this form for any count: paths of 20 siblings take 37 us
// (1000 of them), 0.85 ms (65536) and 3.34 ms (262144) against 368, 1150 and 4211 with
// a thread per path; only paths of one sibling, from 2^17 of them on, are 3 to 6%
// slower.
__global__ void __launch_bounds__(COOP_THREADS) k_root_from_paths_coop(const uint64_t* __restrict__ idx,
                                                                       const uint64_t* __restrict__ leaves,
                                                                       const uint64_t* __restrict__ paths,
                                                                       uint64_t count, uint64_t len,
                                                                       uint64_t* __restrict__ roots) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[COOP_STATES * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    const uint64_t i = (uint64_t)blockIdx.x * COOP_STATES + threadIdx.x / T5C_LANES, q = i < count ? i : count - 1;
    const int w = c.lane % 5;  // the digest word this lane would load
    uint64_t cur = gl_canon(leaves[5 * q + w]);
    uint64_t at = idx[q];
    for (uint64_t k = 0; k < len; k++) {
        const uint64_t sib = paths[(q * len + k) * 5 + w];
        const bool right = at & 1;  // the running digest is the right child
        const uint64_t d = t5c_hash_pair((c.lane < 5) == right ? sib : cur, c);
        cur = __shfl_sync(0xffffffffu, d, (threadIdx.x & 16) + w);
        at >>= 1;
    }
    if (i < count && c.lane < 5) roots[5 * i + c.lane] = cur;
}

// Fiat-Shamir absorb into one device sponge state: the elements (an optional
// leading word `lead`, then data[0..len)), then 1, then zeros to a multiple of
// 10; each 10-word chunk overwrites the rate and is followed by a permutation.
// One warp, both halves on the same state.
__global__ void __launch_bounds__(32) k_sponge_absorb_coop(uint64_t* __restrict__ state,
                                                           const uint64_t* __restrict__ data, uint64_t len,
                                                           int has_lead, uint64_t lead) {
    __shared__ T5CoopTables tables;
    __shared__ double2 xch[2 * 2 * T5_STATE];
    T5Coop c;
    t5c_init(c, tables, xch);
    uint64_t x = gl_to_mont(state[c.lane]);
    const uint64_t total = len + (has_lead ? 1 : 0);
    const uint64_t perms = total / T5_RATE + 1;  // room for the 1
    for (uint64_t k = 0; k < perms; k++) {
        if (c.lane < T5_RATE) {
            const uint64_t j = k * T5_RATE + c.lane;
            uint64_t v = j == total ? 1 : 0;
            if (j < total) v = has_lead ? (j == 0 ? lead : data[j - 1]) : data[j];
            x = gl_to_mont(v);
        }
        t5c_sync();
        x = t5c_permutation(x, c);
    }
    if (threadIdx.x < T5_STATE) state[c.lane] = gl_from_mont(x);
}

namespace {
unsigned blocks_of(uint64_t states) { return (unsigned)((states + COOP_STATES - 1) / COOP_STATES); }
}  // namespace

cudaError_t launch_hash_rows_coop(const uint64_t* table, uint64_t rstride, uint64_t cstride, uint64_t rows,
                                  uint32_t width, uint64_t* digests, uint64_t* tree, int layout, cudaStream_t st) {
    count_launch();
    k_hash_rows_coop<<<blocks_of(rows), COOP_THREADS, 0, st>>>(table, rstride, cstride, rows, width, digests, tree,
                                                               layout);
    return cudaGetLastError();
}

cudaError_t launch_hash_jobs_coop(const HashJobs& jobs, uint32_t blocks, cudaStream_t st) {
    count_launch();
    k_hash_rows_multi_coop<<<blocks, COOP_THREADS, 0, st>>>(jobs);
    return cudaGetLastError();
}
uint64_t coop_blocks(uint64_t rows) { return blocks_of(rows); }

cudaError_t launch_merkle_coop(uint64_t* tree, uint64_t n, uint64_t m, int layout, int levels, cudaStream_t st) {
    count_launch();
    k_merkle_coop<<<(unsigned)coop_tree_blocks(m), COOP_TREE_THREADS, 0, st>>>(tree, n, m, layout, levels);
    return cudaGetLastError();
}

cudaError_t launch_merkle_levels_coop(const LevelJobs& jobs, uint32_t blocks, cudaStream_t st) {
    count_launch();
    k_merkle_levels_coop<<<blocks, COOP_TREE_THREADS, 0, st>>>(jobs);
    return cudaGetLastError();
}

cudaError_t launch_hash_pairs_coop(const uint64_t* left, const uint64_t* right, uint64_t* out, uint64_t count,
                                   cudaStream_t st) {
    count_launch();
    k_hash_pairs_coop<<<blocks_of(count), COOP_THREADS, 0, st>>>(left, right, out, count);
    return cudaGetLastError();
}

cudaError_t launch_tip5_permutations_coop(uint64_t* states, uint64_t count, cudaStream_t st) {
    count_launch();
    k_tip5_perm_coop<<<blocks_of(count), COOP_THREADS, 0, st>>>(states, count);
    return cudaGetLastError();
}

cudaError_t launch_root_from_paths(const uint64_t* idx, const uint64_t* leaves, const uint64_t* paths, uint64_t count,
                                   uint64_t len, uint64_t* roots, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    count_launch();
    k_root_from_paths_coop<<<blocks_of(count), COOP_THREADS, 0, st>>>(idx, leaves, paths, count, len, roots);
    return cudaGetLastError();
}

cudaError_t launch_sponge_absorb(uint64_t* state, const uint64_t* data, uint64_t len, int has_lead, uint64_t lead,
                                 cudaStream_t st) {
    count_launch();
    k_sponge_absorb_coop<<<1, 32, 0, st>>>(state, data, len, has_lead, lead);
    return cudaGetLastError();
}

}  // namespace tvmc
