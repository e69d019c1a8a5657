// K7: the simulations of compute_pvalues drawn on the GPU.
//
// compute_pvalues (src/probability.cpp:376-570) simulates n_sim families
// per root size r = 1..R down the tree (create_family, :351-373, over
// set_weighted_random_family_size, :449-476): every child's size is drawn
// from its parent's matrix row restricted to sizes 0..S-1
// (matrix::select_random_y, src/matrix_cache.cpp:60-66, a
// std::discrete_distribution over the row's first S entries). The
// reference draws from one std::mt19937 in a fixed order, and a family that
// dies out below a node takes fewer draws, so where a family starts in the
// stream hangs on every family before it. Two modes:
//  * the reference's stream. k_mt_words writes its words (one block, ahead of
//    the rest on a stream of its own). k_sim_regular takes 16 root sizes at a
//    time as if no family died out anywhere, and keeps those where none did.
//    For the next one k_sim_len finds for every draw how many draws a family
//    that started there would take (all of them in parallel: about n_nodes times
//    the work of the families themselves, on internal nodes only), and
//    k_sim_chase follows the chain of starts. Then every family is one thread.
//    Words and rounds of launches are the bound; 150,000 families of 12 taxa: a
//    call of 19.8 ms (20.1 with one warp set making and writing the words, 22.4
//    with the chain for every root size, 131 with one host thread drawing).
//  * opt-in, a counter-based generator (the SplitMix64 sequence of Steele, Lea
//    and Flood, OOPSLA 2014, indexed by (family, node)): the same
//    distributions, not the reference's stream, so the p-values agree in
//    distribution, not bit for bit.
//
//  * k_cdf_build: cumulative weights of every (node, parent size) row.
//  * k_sim_draw: one thread per simulated family: sizes in prefix order by
//    inverse-CDF search, the leaf counts, the family's state bound
//    m = min(S, largest + max(50, largest / 5)) (compute_family_probabilities)
//    and its (root size, bound) key.
//  * k_sim_plan (one block): families per key -> offsets, grouped by bound;
//    and 32-family tiles of equal (root size, bound).
//  * k_sim_scatter: the family order.
//  * (k_patterns and k_pat64: families of equal bound share the factor rows of
//    equal subtrees below the root's children.)
//  * k_sim_root: each family's root value from those rows, one state of the
//    root's children only. 150,000 families of 12 taxa, bounds 51 to 170: 19.6
//    ms a call, 75.1 with k_prune64 walking 32-family tiles, which still takes
//    vectors that do not fit a CTA's shared memory and groups whose tables
//    would pass 16 GB. The FP64 pipe is the bound: 10 GFMA over distinct rows,
//    22 without.
//  * k_sort_rows: each root size's n_sim likelihoods sorted (bitonic sort
//    in shared memory), the conditional distributions.
//  * k_pvalue_search: per observed family, the largest share of simulated
//    likelihoods not above its own over root sizes up to 1.25 x its largest
//    count (find_best_pvalue / pvalue, :503-528).
#include "common.cuh"

#include <limits.h>

#include <algorithm>

namespace cafe {
namespace {

constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ull;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Output c + 1 of the SplitMix64 sequence started at `key`, as a double in
// [0, 1) with 53 random bits.
__device__ __forceinline__ double uniform01(uint64_t key, uint64_t c) {
    return (double)(mix64(key + (c + 1) * kGolden) >> 11) * 0x1.0p-53;
}

// The reference's own draws. std::discrete_distribution<int> over a row takes
// two words of the std::mt19937 (generate_canonical: (w0 + 2^32 w1) / 2^64, in
// double) and returns the first size whose cumulative probability, the last
// set to 1, is not below it.
__device__ __forceinline__ double canonical(uint2 w) {
    const double u = ((double)w.x + (double)w.y * 0x1.0p32) * 0x1.0p-64;
    return u < 1.0 ? u : 0x1.fffffffffffffp-1;
}

// (a child's size is near its parent's: the search widens from there)
__device__ __forceinline__ int draw_size(const double* __restrict__ cp, int S, int ps, double u) {
    int lo = 0, hi = S - 1;
    const int g = min(ps, S - 1);
    if (__ldg(cp + g) < u) {
        lo = g + 1;
        int w = 4;
        for (; lo + w < hi && __ldg(cp + lo + w) < u; w *= 2) lo += w + 1;
        hi = min(hi, lo + w);
    } else {
        hi = g;
        int w = 4;
        for (; hi - w > 0 && !(__ldg(cp + hi - w) < u); w *= 2) hi -= w;
        lo = max(0, hi - w);
    }
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(cp + mid) < u) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// MT19937 (Matsumoto and Nishimura, ACM TOMACS 8, 1998), one block: thread i of
// the first half makes words i, i + 227 and i + 454 of each 624, of which the
// later two need only its own earlier ones and the old state; the second half
// tempers and writes the words of the round before.
__device__ __forceinline__ uint32_t mt_twist(uint32_t a, uint32_t b, uint32_t m) {
    const uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
    return m ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}
__device__ __forceinline__ uint32_t mt_temper(uint32_t y) {
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    return y ^ (y >> 18);
}
constexpr int kMtHalf = 256;
__global__ void __launch_bounds__(2 * kMtHalf) k_mt_words(bool first, uint32_t seed, uint32_t* __restrict__ state, int64_t n,
                                                          uint32_t* __restrict__ out) {
    __shared__ uint32_t st[2][kMtWords];
    const bool writer = threadIdx.x >= kMtHalf;
    const int i = threadIdx.x % kMtHalf;
    for (int k = threadIdx.x; !first && k < kMtWords; k += 2 * kMtHalf) st[0][k] = state[k];
    if (first && threadIdx.x == 0) {
        uint32_t x = seed;
        st[0][0] = x;
        for (int k = 1; k < kMtWords; ++k) {
            x = 1812433253u * (x ^ (x >> 30)) + (uint32_t)k;
            st[0][k] = x;
        }
    }
    __syncthreads();
    const int64_t rounds = (n + kMtWords - 1) / kMtWords;
    for (int64_t q = 0; q <= rounds; ++q) {
        const uint32_t* s = st[q & 1];
        uint32_t* t = st[(q & 1) ^ 1];
        if (!writer && i < 227 && q < rounds) {
            const uint32_t x0 = mt_twist(s[i], s[i + 1], s[i + 397]);
            const uint32_t x1 = mt_twist(s[i + 227], s[i + 228], x0);
            t[i] = x0;
            t[i + 227] = x1;
            if (i < 170) {
                const uint32_t nx = i == 169 ? mt_twist(s[0], s[1], s[397]) : s[i + 455];
                t[i + 454] = mt_twist(s[i + 454], nx, x1);
            }
        } else if (writer && q > 0) {
            // (the state the others read now)
            const int64_t left = n - (q - 1) * kMtWords;
            uint32_t* o = out + (q - 1) * kMtWords;
#pragma unroll
            for (int k = i; k < kMtWords; k += kMtHalf)
                if (k < left) o[k] = mt_temper(s[k]);
        }
        __syncthreads();
    }
    for (int k = threadIdx.x; k < kMtWords; k += 2 * kMtHalf) state[k] = st[rounds & 1][k];
}

// A family takes a draw for every node whose parent has genes, so where the
// next one starts depends on its sizes. How many draws the family of root size
// r + 1 that starts at words w takes; sz holds the sizes of the internal nodes
// ([n_internal][kLenThreads], this thread's column).
constexpr int kLenThreads = 128;
__device__ __forceinline__ int draws_of(const SimStreamArgs& a, int r, const uint2* w, int32_t* my) {
    my[a.node_ii[a.root] * kLenThreads] = r + 1;
    int used = 0;
    for (int i = 0; i < a.n_nodes; ++i) {
        const int v = a.prefix[i];
        if (v == a.root) continue;
        const int ps = my[a.node_ii[a.parent[v]] * kLenThreads];
        const int ii = a.node_ii[v];
        if (ii >= 0) my[ii * kLenThreads] = ps > 0 ? draw_size(a.cdf + ((size_t)v * a.n_ps + ps) * a.S, a.S, ps, canonical(w[used])) : 0;
        used += ps > 0;
    }
    return used;
}

// Families that never die out take n - 1 draws each, and from some root size on
// nearly all are such: the families of the next kSpec root sizes (below r_end)
// at the starts they have if they all are. The root sizes before the first
// with another length are done; the last block writes their starts.
constexpr int kSpec = 16;
__global__ void __launch_bounds__(kLenThreads) k_sim_regular(SimStreamArgs a, int r_end) {
    extern __shared__ int32_t sz[];
    __shared__ int last;
    const int r0 = *(volatile int32_t*)&a.state[0], r1 = min(r0 + kSpec, r_end);
    if (r0 >= r_end) return;
    const int most = a.n_nodes - 1;
    const int64_t first = a.starts[(int64_t)r0 * a.n_sim];
    const int64_t t = (int64_t)blockIdx.x * kLenThreads + threadIdx.x;
    if (t < (int64_t)(r1 - r0) * a.n_sim) {
        const int r = r0 + (int)(t / a.n_sim);
        if (draws_of(a, r, a.words + first + t * most, sz + threadIdx.x) != most) atomicMin(&a.state[1], r);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&a.state[2], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int r2 = min(r1, *(volatile int32_t*)&a.state[1]);
    for (int64_t f = threadIdx.x; f <= (int64_t)(r2 - r0) * a.n_sim; f += kLenThreads)
        a.starts[(int64_t)r0 * a.n_sim + f] = first + f * most;
    __syncthreads();
    if (threadIdx.x == 0) {
        a.state[0] = r2;
        a.state[1] = INT_MAX;
        a.state[2] = 0;
        a.state[3] = r2 < r1;
    }
}

// The next root size where some family is not regular: how many draws a family
// takes, for every draw it might start at (n_sim families of at most n - 1 draws
// each).
__global__ void __launch_bounds__(kLenThreads) k_sim_len(SimStreamArgs a) {
    extern __shared__ int32_t sz[];
    if (!a.state[3]) return;
    const int r = a.state[0];
    const int64_t p = (int64_t)blockIdx.x * kLenThreads + threadIdx.x;
    if (p > (int64_t)(a.n_sim - 1) * (a.n_nodes - 1)) return;
    a.len[p] = (uint16_t)draws_of(a, r, a.words + a.starts[(int64_t)r * a.n_sim] + p, sz + threadIdx.x);
}

// The chain of starts through those lengths, one block: jumps over eight
// families by doubling, one thread along them, then a thread per eight.
constexpr int kChasePos = 24576;          // starts in shared memory (at least 32 x (kMaxNodes - 1))
constexpr int kChaseThreads = 1024;
static_assert(kChasePos >= 32 * (kMaxNodes - 1), "a segment holds 32 families");
__global__ void __launch_bounds__(kChaseThreads) k_sim_chase(SimStreamArgs a) {
    extern __shared__ uint16_t jump[];    // [3][kChasePos]
    if (!a.state[3]) return;
    const int r = a.state[0];
    __shared__ int32_t eighth[kChasePos / 8 + 1];
    uint16_t* one = jump;
    const int tid = threadIdx.x, most = a.n_nodes - 1;
    const int seg = (kChasePos / most) & ~31;
    int64_t* starts = a.starts + (int64_t)r * a.n_sim;
    int64_t at = 0;                       // relative to the root size's first draw
    const int64_t first = starts[0];
    for (int k0 = 0; k0 < a.n_sim; k0 += seg) {
        const int q = min(seg, a.n_sim - k0), P = (q - 1) * most + 1;
        for (int p = tid; p < P; p += kChaseThreads) {
            // (past the last family's last possible start: not on the chain)
            const int64_t g = at + p;
            one[p] = g <= (int64_t)(a.n_sim - 1) * most ? a.len[g] : 0;
        }
        __syncthreads();
        const uint16_t* src = one;
        for (int d = 0; d < 3; ++d) {
            uint16_t* dst = jump + (1 + (d & 1)) * kChasePos;
            for (int p = tid; p < P; p += kChaseThreads) {
                const int j = src[p], n = p + j;
                dst[p] = n < P ? (uint16_t)(j + src[n]) : 0;
            }
            __syncthreads();
            src = dst;
        }
        const int n8 = (q + 7) / 8;
        if (tid == 0) {
            int p = 0;
            for (int g = 0; g < n8; ++g) {
                eighth[g] = p;
                if (g + 1 < n8) p += src[p];
            }
        }
        __syncthreads();
        for (int g = tid; g < n8; g += kChaseThreads) {
            int p = eighth[g];
            const int k1 = min(8 * g + 8, q);
            for (int k = 8 * g; k < k1; ++k) {
                starts[k0 + k] = first + at + p;
                p += one[p];
            }
            if (g == n8 - 1) starts[k0 + q] = first + at + p;
        }
        __syncthreads();
        at = starts[k0 + q] - first;
    }
    if (tid == 0) {
        a.state[0] = r + 1;
        a.state[3] = 0;
    }
}

template <bool NORM>
__global__ void __launch_bounds__(128) k_cdf_build(const double* const* __restrict__ mats, int n_nodes, int msize,
                                                   int S, int n_ps, double* __restrict__ cdf) {
    const int v = blockIdx.x;
    const int ps = blockIdx.y * blockDim.x + threadIdx.x;
    if (v >= n_nodes || ps >= n_ps) return;
    const double* M = mats[v];
    if (!M) return;   // the root
    const double* row = M + (size_t)ps * msize;
    double* out = cdf + ((size_t)v * n_ps + ps) * S;
    double acc = 0.0;
    if (NORM) {
        double sum = 0.0;
        for (int c = 0; c < S; ++c) sum += row[c];
        for (int c = 0; c < S; ++c) {
            acc += row[c] / sum;
            out[c] = c + 1 < S ? acc : 1.0;
        }
        return;
    }
    for (int c = 0; c < S; ++c) {
        acc += row[c];
        out[c] = acc;
    }
}

template <bool STREAM>
__global__ void __launch_bounds__(128) k_sim_draw(SimDrawArgs a) {
    const int64_t fi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (fi >= a.n_families) return;
    const int r = (int)(fi / a.n_sim);     // root size r + 1
    int32_t* sz = a.sizes + (size_t)fi * a.n_nodes;
    sz[a.root] = r + 1;
    int mx = r + 1;
    const int S = a.S;
    const uint2* w = STREAM ? a.words + a.starts[fi] : nullptr;
    for (int i = 0; i < a.n_nodes; ++i) {
        const int v = a.prefix[i];
        if (v == a.root) continue;
        const int ps = sz[a.parent[v]];
        int c = 0;
        const double* cd = a.cdf + ((size_t)v * a.n_ps + ps) * S;
        if (STREAM && ps > 0) {
            c = draw_size(cd, S, ps, canonical(*w++));
        } else if (ps > 0) {
            const double total = cd[S - 1];
            if (total > 0.0) {
                // first size whose cumulative weight exceeds u * total
                double target = uniform01(a.key, (uint64_t)fi * a.n_nodes + v) * total;
                if (target >= total) target = nextafter(total, 0.0);
                int lo = 0, hi = S - 1;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (cd[mid] > target) hi = mid;
                    else lo = mid + 1;
                }
                c = lo;
            }
        }
        sz[v] = c;
        mx = max(mx, c);
        if (a.leaf_col[v] >= 0) a.counts[(size_t)fi * a.n_leaves + a.leaf_col[v]] = c;
    }
    const int m = min(S, mx + max(50, mx / 5));
    const int key = m * a.R + r;
    a.keys[fi] = key;
    atomicAdd(&a.hist[key], 1);
}

// Block-wide inclusive sum of one value per thread (1024 threads).
__device__ __forceinline__ int64_t block_scan(int64_t x, int64_t* sh, int64_t* total) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int64_t w = sh[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sh[lane] = w;
    }
    __syncthreads();
    if (warp > 0) x += sh[warp - 1];
    *total = sh[31];
    __syncthreads();
    return x;
}

__global__ void __launch_bounds__(1024) k_sim_plan(SimPlanArgs a) {
    __shared__ int64_t sh[32];
    int64_t fam_base = 0, tile_base = 0;
    const int n_keys = (a.S + 1) * a.R;
    for (int k0 = 0; k0 < n_keys; k0 += 1024) {
        const int key = k0 + threadIdx.x;
        const int64_t cnt = key < n_keys ? a.hist[key] : 0;
        const int64_t nt = (cnt + 31) / 32;
        int64_t tf, tt;
        const int64_t fam_inc = block_scan(cnt, sh, &tf);
        const int64_t tile_inc = block_scan(nt, sh, &tt);
        if (key < n_keys) {
            const int64_t f0 = fam_base + fam_inc - cnt, t0 = tile_base + tile_inc - nt;
            a.cursor[key] = (int32_t)f0;
            const int m = key / a.R, r = key % a.R;
            if (r == 0) a.bound_first[m] = f0;
            for (int64_t i = 0; i < nt && t0 + i < a.max_tiles; ++i) {
                PruneTile t{};
                t.first = (int)(f0 + 32 * i);
                t.count = (int)(cnt - 32 * i < 32 ? cnt - 32 * i : 32);
                t.k = 0;
                t.S = m;
                t.R = 1;
                t.root_lo = r + 1;
                a.tiles[t0 + i] = t;
            }
        }
        fam_base += tf;
        tile_base += tt;
    }
    if (threadIdx.x == 0) a.bound_first[a.S + 1] = fam_base;
    if (threadIdx.x == 0) *a.n_tiles = (int32_t)(tile_base < a.max_tiles ? tile_base : a.max_tiles);
}

__global__ void __launch_bounds__(256) k_sim_scatter(const int32_t* __restrict__ keys, int64_t n,
                                                     int32_t* __restrict__ cursor, int64_t* __restrict__ perm) {
    const int64_t fi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (fi >= n) return;
    const int pos = atomicAdd(&cursor[keys[fi]], 1);
    perm[pos] = fi;
}

// Four lanes per family, one FMA chain each (columns 0, 1, 2, 3 mod 4, as
// every FP64 sum here): the one state of each root child's factor that the
// family's root size needs.
__global__ void __launch_bounds__(256) k_sim_root(SimRootArgs a) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t i = min(a.i0 + (t >> 2), a.i1 - 1);      // (past the last: the last again)
    const int h = (int)(t & 3);
    const TreePlan& P = a.plan;
    const int64_t f = a.perm[i];
    const int key = a.keys[f], m = key / a.R, r = key % a.R + 1;
    const int pitch = (m + 2) & ~1;
    auto row = [&](int ch) -> const double* {      // the factor row of grandchild ch
        const int64_t at = a.tab[(size_t)m * P.n_nodes + ch];
        const int lc = P.leaf_col[ch];
        if (lc >= 0) return a.table + at + (int64_t)a.counts[(size_t)f * P.n_leaves + lc] * a.leaf_pitch;
        const int ii = a.node_ii[ch];
        const int64_t idx = a.num[(size_t)ii * a.F + a.rep[(size_t)ii * a.F + i]] - a.base[(size_t)ii * (a.n_groups + 1) + m];
        return a.table + at + idx * pitch;
    };
    double value = 1.0;
    const int ri = P.n_internal - 1;               // the root
    for (int c = P.cstart[ri]; c < P.cstart[ri + 1]; ++c) {
        const int ch = P.child[c];
        const double* M = a.mats[ch] + (size_t)r * a.ld_mat;
        const int lc = P.leaf_col[ch];
        if (lc >= 0) {
            value *= M[a.counts[(size_t)f * P.n_leaves + lc]];
            continue;
        }
        const int ii = a.node_ii[ch], g0 = P.cstart[ii], g1 = P.cstart[ii + 1];
        const double* p0 = row(P.child[g0]);
        const double* p1 = g1 - g0 > 1 ? row(P.child[g0 + 1]) : nullptr;
        double acc = 0.0;
#pragma unroll 4
        for (int j = h; j <= m; j += 4) {
            double u = p0[j];
            if (p1) u *= p1[j];
            for (int g = g0 + 2; g < g1; ++g) u *= row(P.child[g])[j];
            acc = fma(M[j], u, acc);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        value *= acc;
    }
    if (h == 0 && a.i0 + (t >> 2) < a.i1) a.out[f] = value;
}

// One block per row of n values: ascending bitonic sort of the row padded
// with +inf to P = a power of two (dynamic shared memory, P doubles).
__global__ void __launch_bounds__(512) k_sort_rows(double* __restrict__ v, int n, int P) {
    extern __shared__ double s[];
    double* row = v + (size_t)blockIdx.x * n;
    for (int i = threadIdx.x; i < P; i += blockDim.x) s[i] = i < n ? row[i] : INFINITY;
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < P; i += blockDim.x) {
                const int l = i ^ j;
                if (l > i) {
                    const bool up = (i & k) == 0;
                    const double x = s[i], y = s[l];
                    if (up ? (x > y) : (x < y)) {
                        s[i] = y;
                        s[l] = x;
                    }
                }
            }
            __syncthreads();
        }
    for (int i = threadIdx.x; i < n; i += blockDim.x) row[i] = s[i];
}

__global__ void __launch_bounds__(128) k_pvalue_search(PvalueSearchArgs a) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.F) return;
    int largest = 0;
    for (int c = 0; c < a.n_leaves; ++c) largest = max(largest, a.counts[(size_t)f * a.n_leaves + c]);
    const int check = min(a.R, (int)rint(largest * 1.25));
    double best = 0.0;
    for (int j = 0; j < check; ++j) {
        const double v = a.obs[(size_t)f * a.R + j];
        const double* d = a.sorted + (size_t)j * a.n_sim;
        // first simulated value above v (the reference's upper_bound; past
        // the end it counts n_sim - 1)
        int lo = 0, hi = a.n_sim;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (d[mid] > v) hi = mid;
            else lo = mid + 1;
        }
        const int idx = lo == a.n_sim ? a.n_sim - 1 : lo;
        best = fmax(best, idx / (double)a.n_sim);
    }
    a.out[f] = best;
}

}  // namespace

uint64_t sim_seed_key(uint32_t seed) {
    uint64_t z = (uint64_t)seed + kGolden;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

cudaError_t pvalue_kernels_init() {
    cudaError_t e = cudaFuncSetAttribute(k_sort_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortRowsMaxP * 8);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sim_chase, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * kChasePos * (int)sizeof(uint16_t));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sim_len, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kMaxNodes * kLenThreads / 2 * (int)sizeof(int32_t));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sim_regular, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kMaxNodes * kLenThreads / 2 * (int)sizeof(int32_t));
    return e;
}

cudaError_t launch_cdf_build(const double* const* mats, int n_nodes, int msize, int S, int n_ps, bool normalised,
                             double* cdf, cudaStream_t s) {
    if (n_nodes <= 0 || n_ps <= 0 || S <= 0) return cudaSuccess;
    const dim3 grid((unsigned)n_nodes, (unsigned)((n_ps + 127) / 128));
    if (normalised) k_cdf_build<true><<<grid, 128, 0, s>>>(mats, n_nodes, msize, S, n_ps, cdf);
    else k_cdf_build<false><<<grid, 128, 0, s>>>(mats, n_nodes, msize, S, n_ps, cdf);
    return cudaGetLastError();
}

cudaError_t launch_mt_words(bool first, uint32_t seed, uint32_t* state, int64_t n, uint32_t* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_mt_words<<<1, 2 * kMtHalf, 0, s>>>(first, seed, state, n, out);
    return cudaGetLastError();
}

cudaError_t launch_sim_starts(const SimStreamArgs& a, int r0, int r1, cudaStream_t s) {
    const int64_t P = (int64_t)(a.n_sim - 1) * (a.n_nodes - 1) + 1;
    const size_t smem = (size_t)a.n_internal * kLenThreads * sizeof(int32_t);
    const auto blocks = [](int64_t n) { return (unsigned)((n + kLenThreads - 1) / kLenThreads); };
    // (a round does at least one root size; the rounds left over find none)
    for (int r = r0; r < r1; ++r) {
        k_sim_regular<<<blocks((int64_t)kSpec * a.n_sim), kLenThreads, smem, s>>>(a, r1);
        k_sim_len<<<blocks(P), kLenThreads, smem, s>>>(a);
        k_sim_chase<<<1, kChaseThreads, 3 * kChasePos * sizeof(uint16_t), s>>>(a);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_sim_draw(const SimDrawArgs& a, cudaStream_t s) {
    if (a.n_families <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((a.n_families + 127) / 128);
    if (a.starts) k_sim_draw<true><<<grid, 128, 0, s>>>(a);
    else k_sim_draw<false><<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sim_plan(const SimPlanArgs& a, cudaStream_t s) {
    k_sim_plan<<<1, 1024, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sim_root(const SimRootArgs& a, cudaStream_t s) {
    if (a.i1 <= a.i0) return cudaSuccess;
    k_sim_root<<<(unsigned)((4 * (a.i1 - a.i0) + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sim_scatter(const int32_t* keys, int64_t n, int32_t* cursor, int64_t* perm, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_sim_scatter<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(keys, n, cursor, perm);
    return cudaGetLastError();
}

cudaError_t launch_sort_rows(double* v, int rows, int n, cudaStream_t s) {
    if (rows <= 0 || n <= 0) return cudaSuccess;
    int P = 1;
    while (P < n) P <<= 1;
    if (P > kSortRowsMaxP) return cudaErrorInvalidValue;
    k_sort_rows<<<(unsigned)rows, 512, (size_t)P * sizeof(double), s>>>(v, n, P);
    return cudaGetLastError();
}

cudaError_t launch_pvalue_search(const PvalueSearchArgs& a, cudaStream_t s) {
    if (a.F <= 0) return cudaSuccess;
    k_pvalue_search<<<(unsigned)((a.F + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace cafe
