// LDE of short columns (N <= 2^11): whole columns per CTA.
#include <algorithm>

#include "ntt_sub.cuh"

namespace tvmc {

// T = 2^lT columns: the inverse transform of the columns, then the forward
// transforms of 2^lc cosets of every column at a time (sequence u = t * 2^lc + c),
// so that a short column's cosets fill the CTA together and an output row of
// cosets is written as one run.  One coset at a time left three quarters of the
// threads idle: 2^8 x 379, x4, 43 -> 26 us.  ONE: no expansion, le = lc = 0, where
// the index arithmetic of cosets is dead weight (2^8 x 379 14.5 us with it, 12.5
// without; 2^10 x 379 74 and 71).
template <int LS, bool ONE>
__global__ void __launch_bounds__(NTT_THREADS) k_lde_small(const uint64_t* trace, uint64_t tld, uint64_t* out,
                                                           uint64_t old, uint64_t cols, int lT, int le_arg,
                                                           int lc_arg, const uint64_t* tw12_f, const uint64_t* sc_lo,
                                                           const uint64_t* sc_hi, int hi_len, const uint64_t* add,
                                                           int rm) {
    extern __shared__ uint64_t sm[];
    constexpr int n = 1 << LS;
    const int le = ONE ? 0 : le_arg, lc = ONE ? 0 : lc_arg;
    const int E = 1 << le, EC = 1 << lc;
    uint64_t* twf = sm;                    // forward root only (the inverse negates its input index)
    uint64_t* cf = twf + n;                // coefficients (natural order)
    uint64_t* s = cf + spad_words(n, lT);  // transposes
    load_tw<LS>(twf, tw12_f);
    __syncthreads();
    const uint64_t c0 = (uint64_t)blockIdx.x << lT;
    sub_dft<LS>(  // inverse: forward DFT of the index-negated column
        s, lT, twf,
        [&](int k, int t) { return c0 + t < cols ? gl_canon(trace[(c0 + t) * tld + (-k & (n - 1))]) : 0ull; },
        [&](int k, int t, uint64_t v) { cf[spos(k, lT) + t] = v; });
    __syncthreads();
    for (int cb = 0; cb < E; cb += EC) {
        sub_dft<LS>(
            s, lT + lc, twf,
            [&](int k, int u) {
                const int t = u >> lc, c = cb + (u & (EC - 1));
                uint64_t x = cf[spos(k, lT) + t];
                if (rm && k < rm && c0 + t < cols) x = gl_add_pc(x, add[((c0 + t) * E + c) * rm + k]);
                return gl_mul_c(x, tw2(sc_lo + 4096 * c, sc_hi + hi_len * c, (uint32_t)k));
            },
            [&](int q, int u, uint64_t v) {
                const int t = u >> lc;
                if (c0 + t < cols) out[(c0 + t) * old + (uint64_t)q * E + cb + (u & (EC - 1))] = v;
            });
        __syncthreads();
    }
}

cudaError_t launch_lde_small(const LdePlan& pl, const uint64_t* trace, uint64_t tld, uint64_t* out, uint64_t old,
                             uint64_t cols, const uint64_t* add, int rm, cudaStream_t st) {
    const int l = pl.logn, le = pl.log_exp;
    const int hi_len = l > 12 ? (1 << (l - 12)) : 1;
    const int lT = std::clamp(10 - l, 0, l <= 5 ? 8 : 3);  // about 2^10 words of coefficients per CTA
    const int lc = le < 2 ? le : 2;  // four cosets at a time: 100 KB at 2^11
    const int T = 1 << lT;
    const size_t smem = words_bytes((size_t)(1u << l) + spad_words(1 << l, lT) + spad_words(1 << l, lT + lc));
    return dispatch_ls(l, [&]<int LS>() -> cudaError_t {
        auto kern = le ? k_lde_small<LS, false> : k_lde_small<LS, true>;
        cudaError_t e = set_smem((const void*)kern, smem);
        if (e != cudaSuccess) return e;
        count_launch();
        kern<<<(unsigned)((cols + T - 1) / T), NTT_THREADS, smem, st>>>(
            trace, tld, out, old, cols, lT, le, lc, pl.tw12_f, pl.sc_lo, pl.sc_hi, hi_len, add, rm);
        return cudaGetLastError();
    });
}

}  // namespace tvmc
