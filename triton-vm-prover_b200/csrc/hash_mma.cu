// Tip5 row hashing and wide Merkle levels on the tensor-core permutation
// (tip5_mma.cuh).
//
// Two threads per sponge state; a group of 256 threads takes tiles of 128 rows,
// and four groups (one CTA of 1024 threads) fill an SM.  A CTA ends after a bounded
// number of tiles (TileSpan), so that kernels of other streams get in.  Rows are
// read column-major (a warp reads 32 consecutive rows of one column, 256
// contiguous bytes).  Semantics:
// Tip5::hash_varlen (src/hash/tip5.cpp:246-282) -- zero state, overwrite the
// rate with each full chunk and permute, last chunk = rest, 1, zeros.
#include "hash_mma.h"
#include "internal.cuh"
#include "tip5_mma.cuh"

namespace tvmc {

namespace {

extern __shared__ uint8_t t5m_smem[];

__device__ __forceinline__ uint32_t dyn_base() { return (uint32_t)__cvta_generic_to_shared(t5m_smem); }

__device__ __forceinline__ void mark_dead(const T5Mma& c, uint64_t* status) {
    if (c.waits.dead && status) *status = 1;
}

// Absorbs `perms` chunks of the row at p (element i at p[i * cs]): its n
// elements, then 1 and zeros.  Only the chunk that holds the end tests its words.
__device__ __forceinline__ void absorb(uint64_t (&s)[T5M_WORDS], const uint64_t* __restrict__ p, uint64_t cs,
                                       uint32_t perms, uint32_t n, T5Mma& c) {
    static_assert(T5M_PARTS == 2 && T5_RATE == 10, "part 0 holds rate words 0, 1, 4..9, part 1 words 2, 3");
    const uint64_t* p0 = p + (uint64_t)(T5M_LOOKUPS * c.part) * cs;
    const uint64_t* p1 = p + 4 * cs;
    for (uint32_t k = 0; k < perms; k++) {
        if ((k + 1) * T5_RATE <= n) {
#pragma unroll
            for (int i = 0; i < T5M_LOOKUPS; i++) s[i] = gl_to_mont(__ldg(p0 + i * cs));
            if (c.part == 0) {
#pragma unroll
                for (int i = 0; i < T5_RATE - 4; i++) s[T5M_LOOKUPS + i] = gl_to_mont(__ldg(p1 + i * cs));
            }
            p0 += T5_RATE * cs;
            p1 += T5_RATE * cs;
        } else {
#pragma unroll
            for (int i = 0; i < T5M_WORDS; i++) {
                const uint32_t w = t5m_word(c.part, i), j = k * T5_RATE + w;
                if (w < T5_RATE) s[i] = j < n ? gl_to_mont(__ldg(p + (uint64_t)j * cs)) : (j == n ? T5_MONT_ONE : 0);
            }
        }
        t5m_permutation(s, c);
    }
}

__device__ __forceinline__ void zero(uint64_t (&s)[T5M_WORDS]) {
#pragma unroll
    for (int i = 0; i < T5M_WORDS; i++) s[i] = 0;
}

// The digest of a squeezed state: words 0-4.
__device__ __forceinline__ void store_digest(const uint64_t (&s)[T5M_WORDS], uint64_t* p, const T5Mma& c) {
#pragma unroll
    for (int i = 0; i < T5M_LOOKUPS + 1; i++) {
        const int w = t5m_word(c.part, i);
        if (w < 5) p[w] = gl_from_mont(s[i]);
    }
}

// hash_pair of the plain digests at l and r.
__device__ __forceinline__ void pair_hash(uint64_t (&s)[T5M_WORDS], const uint64_t* l, const uint64_t* r, T5Mma& c) {
#pragma unroll
    for (int i = 0; i < T5M_WORDS; i++) {
        const int w = t5m_word(c.part, i);
        s[i] = w < T5_RATE ? gl_to_mont(w < 5 ? l[w] : r[w - 5]) : T5_MONT_ONE;
    }
    t5m_permutation(s, c);
}

// How a launch's tiles go to its CTAs.  The CTAs form rounds of `ctas` (one per
// SM); a round takes ctas * T5M_GROUPS * depth tiles, tile i of it by group
// (i / ctas) mod T5M_GROUPS of CTA i mod ctas, so that a last, partial round is
// spread over all SMs.
struct TileSpan {
    uint32_t tiles, ctas, depth;
};
// Permutations of a group before its CTA ends, 21 us each with all four groups at
// work.  A CTA holds its SM's registers and shared memory until then, and only then
// is a kernel of a greater-priority stream (an opening, a small request) dispatched
// there.  Against the commit of 2^20 x 379 (x4), an opening took at most 43 ms with
// one CTA per SM for the whole launch, 1.6 ms with 76 permutations and 1.0 with 38
// (a commit of 2^10 x 379: 44, 4.9 and 2.7 ms); the row hash of 262144 x 379 took
// 2.85, 2.91 and 2.92 ms in one build of each (a CTA's table fill is 8 us).
constexpr uint32_t CTA_PERMS = 38;
TileSpan tile_span(uint64_t tiles, uint64_t perms_per_tile, int sms) {
    const uint32_t depth = (uint32_t)(CTA_PERMS / perms_per_tile);
    return TileSpan{(uint32_t)tiles, (uint32_t)(tiles < (uint64_t)sms ? tiles : (uint64_t)sms), depth ? depth : 1};
}
uint32_t span_ctas(const TileSpan& s) {
    const uint64_t round = (uint64_t)s.ctas * T5M_GROUPS * s.depth, rest = s.tiles % round;
    return (uint32_t)(s.tiles / round * s.ctas + (rest < s.ctas ? rest : s.ctas));
}

// The tiles of this thread's group.  Each is formed anew from the block index: kept
// across the permutations, the loop's bounds cost registers and 2% of the row hash.
template <class F>
__device__ __forceinline__ void for_tiles(const T5Mma& c, const TileSpan& s, F&& body) {
    for (uint32_t k = 0; k < s.depth; k++) {
        const uint32_t t = (blockIdx.x / s.ctas * s.depth + k) * (s.ctas * T5M_GROUPS) + blockIdx.x % s.ctas +
                           s.ctas * c.group;
        if (t >= s.tiles) break;
        body((uint64_t)t);
    }
}

}  // namespace

// Leaf digests of `rows` rows, element (r, c) at tab[r * rstride + c * cstride], to
// consecutive slots (the leaves of a tree are, in either layout).
__global__ void __launch_bounds__(T5M_THREADS, 1) k_hash_rows_mma(const uint64_t* __restrict__ tab, uint64_t rstride,
                                                                  uint64_t cstride, uint64_t rows, uint32_t width,
                                                                  uint64_t* __restrict__ leaves,
                                                                  uint64_t* status, TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        const uint64_t row = tile * T5M_STATES + c.row;
        const bool live = row < rows;
        uint64_t s[T5M_WORDS];
        zero(s);
        absorb(s, tab + (live ? row : 0) * rstride, cstride, width / T5_RATE + 1, width, c);
        if (live) store_digest(s, leaves + 5 * row, c);
    });
    mark_dead(c, status);
    t5m_done(c);
}

// The same for up to HASH_MULTI_MAX tables: tile i belongs to the job j with
// block0[j] <= i < block0[j + 1].
__global__ void __launch_bounds__(T5M_THREADS, 1) k_hash_rows_multi_mma(const __grid_constant__ HashJobs jobs,
                                                                        TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        int j = 0;
        for (int k = 1; k < jobs.count; k++)
            if (jobs.j[k].block0 <= tile) j = k;
        const uint64_t L = jobs.j[j].L;
        const uint32_t width = jobs.j[j].width;
        const uint64_t row = (tile - jobs.j[j].block0) * T5M_STATES + c.row;
        const bool live = row < L;
        uint64_t s[T5M_WORDS];
        zero(s);
        absorb(s, jobs.j[j].lde + (live ? row : 0), L, width / T5_RATE + 1, width, c);
        if (live) store_digest(s, jobs.j[j].tree + 5 * (L + row), c);
        mark_dead(c, jobs.j[j].tree);
    });
    t5m_done(c);
}

// Frugal streaming: absorb one stripe of `ncols` LDE columns (column-major,
// stride L) into the sponge of every row.  Between stripes only the capacity
// words 10..15 survive (overwrite mode replaces the rate at every absorb), so
// they are all that is stored: cap[w*L + r], w < 6 (coalesced per word).  The
// first stripe starts from the zero state.  Every stripe but the last must hold
// whole 10-column chunks; the last one appends the hash_varlen padding (rest, 1,
// zeros), finishes the digest and writes it as leaf r of the heap tree.
__global__ void __launch_bounds__(T5M_THREADS, 1) k_absorb_stripe_mma(const uint64_t* __restrict__ stripe, uint64_t L,
                                                                      uint32_t ncols, uint64_t* __restrict__ cap,
                                                                      int first, int last,
                                                                      uint64_t* __restrict__ tree, TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        const uint64_t row = tile * T5M_STATES + c.row;
        const bool live = row < L;
        uint64_t s[T5M_WORDS];
#pragma unroll
        for (int i = 0; i < T5M_WORDS; i++) {
            const int w = t5m_word(c.part, i) - T5_RATE;
            s[i] = w >= 0 && !first && live ? cap[(uint64_t)w * L + row] : 0;
        }
        absorb(s, stripe + (live ? row : 0), L, ncols / T5_RATE + (last ? 1 : 0), ncols, c);
        if (!live) return;
        if (last) {
            store_digest(s, tree + 5 * (L + row), c);
            return;
        }
#pragma unroll
        for (int i = 0; i < T5M_WORDS; i++) {
            const int w = t5m_word(c.part, i) - T5_RATE;
            if (w >= 0) cap[(uint64_t)w * L + row] = s[i];
        }
    });
    mark_dead(c, tree);
    t5m_done(c);
}

// One tree level: parent p in [m/2, m) = hash_pair(node 2p, node 2p + 1).
__global__ void __launch_bounds__(T5M_THREADS, 1) k_merkle_level_mma(uint64_t* __restrict__ tree, uint64_t n,
                                                                     uint64_t m, int layout, uint64_t* status,
                                                                     TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    const uint64_t parents = m >> 1;
    for_tiles(c, span, [&](uint64_t tile) {
        const uint64_t i = tile * T5M_STATES + c.row;
        const bool live = i < parents;
        const uint64_t par = parents + (live ? i : 0);
        uint64_t s[T5M_WORDS];
        pair_hash(s, tree + 5 * node_slot(2 * par, n, layout), tree + 5 * node_slot(2 * par + 1, n, layout), c);
        if (live) store_digest(s, tree + 5 * node_slot(par, n, layout), c);
    });
    mark_dead(c, status);
    t5m_done(c);
}

// The same for up to HASH_MULTI_MAX heap trees; tiles as in k_hash_rows_multi_mma.
__global__ void __launch_bounds__(T5M_THREADS, 1) k_merkle_levels_mma(const __grid_constant__ LevelJobs jobs,
                                                                      TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        int j = 0;
        for (int k = 1; k < jobs.count; k++)
            if (jobs.j[k].block0 <= tile) j = k;
        uint64_t* tree = jobs.j[j].tree;
        const uint64_t parents = jobs.j[j].m >> 1, i = (tile - jobs.j[j].block0) * T5M_STATES + c.row;
        const bool live = i < parents;
        const uint64_t par = parents + (live ? i : 0);
        uint64_t s[T5M_WORDS];
        pair_hash(s, tree + 10 * par, tree + 10 * par + 5, c);
        if (live) store_digest(s, tree + 5 * par, c);
        mark_dead(c, tree);
    });
    t5m_done(c);
}

__global__ void __launch_bounds__(T5M_THREADS, 1) k_hash_pairs_mma(const uint64_t* __restrict__ left,
                                                                   const uint64_t* __restrict__ right,
                                                                   uint64_t* __restrict__ out, uint64_t count,
                                                                   uint64_t* status, TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        const uint64_t i = tile * T5M_STATES + c.row, k = i < count ? i : 0;
        uint64_t s[T5M_WORDS];
        pair_hash(s, left + 5 * k, right + 5 * k, c);
        if (i < count) store_digest(s, out + 5 * i, c);
    });
    mark_dead(c, status);
    t5m_done(c);
}

// A part's words lie in aligned pairs of the state; `pairs`: the array is aligned
// for 16-byte accesses (131072 states 57.6 us by single words, 50.4 by pairs; the
// thread-per-state kernel before these took 53.6).
__global__ void __launch_bounds__(T5M_THREADS, 1) k_tip5_perm_mma(uint64_t* __restrict__ states, uint64_t count,
                                                                  bool pairs, uint64_t* status, TileSpan span) {
    T5Mma c;
    t5m_init(c, dyn_base());
    for_tiles(c, span, [&](uint64_t tile) {
        const uint64_t i = tile * T5M_STATES + c.row;
        const bool live = i < count;
        uint64_t s[T5M_WORDS];
        zero(s);
        if (live && pairs) {
#pragma unroll
            for (int k = 0; k < T5M_WORDS; k += 2) {
                const ulonglong2 w = *(const ulonglong2*)(states + T5_STATE * i + t5m_word(c.part, k));
                s[k] = gl_to_mont(w.x);
                s[k + 1] = gl_to_mont(w.y);
            }
        } else if (live) {
#pragma unroll
            for (int k = 0; k < T5M_WORDS; k++) s[k] = gl_to_mont(states[T5_STATE * i + t5m_word(c.part, k)]);
        }
        t5m_permutation(s, c);
        if (live && pairs) {
#pragma unroll
            for (int k = 0; k < T5M_WORDS; k += 2)
                *(ulonglong2*)(states + T5_STATE * i + t5m_word(c.part, k)) =
                    make_ulonglong2(gl_from_mont(s[k]), gl_from_mont(s[k + 1]));
        } else if (live) {
#pragma unroll
            for (int k = 0; k < T5M_WORDS; k++) states[T5_STATE * i + t5m_word(c.part, k)] = gl_from_mont(s[k]);
        }
    });
    mark_dead(c, status);
    t5m_done(c);
}

namespace {

// kern(args..., span) over tiles of perms permutations each; status: the (first)
// word it reports to.
template <class... P, class... A>
cudaError_t launch(void (*kern)(P...), uint64_t tiles, uint64_t perms, cudaStream_t st, uint64_t* status, A... args) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = raise_smem_limit((const void*)kern);
    if (e != cudaSuccess) return e;
    const TileSpan span = tile_span(tiles, perms, sms);
    count_launch();
    kern<<<span_ctas(span), T5M_THREADS, T5M_BYTES, st>>>(args..., span);
    return mma_launched(status, st);
}

}  // namespace

uint64_t mma_tiles(uint64_t rows) { return (rows + T5M_STATES - 1) / T5M_STATES; }

cudaError_t launch_hash_rows_mma(const uint64_t* table, uint64_t rstride, uint64_t cstride, uint64_t rows,
                                 uint32_t width, uint64_t* digests, uint64_t* tree, int layout, cudaStream_t st,
                                 uint64_t* status) {
    return launch(k_hash_rows_mma, mma_tiles(rows), width / T5_RATE + 1, st, status, table, rstride, cstride, rows, width,
                  tree ? tree + 5 * node_slot(rows, rows, layout) : digests, status);
}

cudaError_t launch_hash_jobs_mma(const HashJobs& jobs, uint32_t tiles, cudaStream_t st) {
    uint32_t width = 0;
    for (int k = 0; k < jobs.count; k++) width = jobs.j[k].width > width ? jobs.j[k].width : width;
    return launch(k_hash_rows_multi_mma, tiles, width / T5_RATE + 1, st, jobs.j[0].tree, jobs);
}

cudaError_t launch_absorb_stripe_mma(const uint64_t* stripe, uint64_t L, uint32_t ncols, uint64_t* cap, int first,
                                     int last, uint64_t* tree, cudaStream_t st) {
    return launch(k_absorb_stripe_mma, mma_tiles(L), ncols / T5_RATE + 1, st, tree, stripe, L, ncols, cap, first, last, tree);
}

cudaError_t launch_merkle_level_mma(uint64_t* tree, uint64_t n, uint64_t m, int layout, cudaStream_t st,
                                    uint64_t* status) {
    return launch(k_merkle_level_mma, mma_tiles(m >> 1), 1, st, status, tree, n, m, layout, status);
}

cudaError_t launch_merkle_levels_mma(const LevelJobs& jobs, uint32_t tiles, cudaStream_t st) {
    return launch(k_merkle_levels_mma, tiles, 1, st, jobs.j[0].tree, jobs);
}

cudaError_t launch_hash_pairs_mma(const uint64_t* left, const uint64_t* right, uint64_t* out, uint64_t count,
                                  cudaStream_t st, uint64_t* status) {
    return launch(k_hash_pairs_mma, mma_tiles(count), 1, st, status, left, right, out, count, status);
}

cudaError_t launch_tip5_permutations_mma(uint64_t* states, uint64_t count, cudaStream_t st, uint64_t* status) {
    return launch(k_tip5_perm_mma, mma_tiles(count), 1, st, status, states, count,
                  reinterpret_cast<uintptr_t>(states) % 16 == 0, status);
}

unsigned int mma_timeouts() {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_mma8_timeouts, sizeof v);
    return v;
}

}  // namespace tvmc
