// FP64 recompute of the category terms a mixed-precision pass left open: the
// arithmetic of k_prune64 in its scaled mode, for single (family, category)
// terms spread over the chip.
//
// Few terms are flagged (often one or two of tens of thousands), and a term's
// walk up the tree is serial, so what bounds it is latency: one SM's FP64 pipe
// (two FMAs a clock) needs 50 us for the 200,000 products of a 96-state walk of
// 24 taxa and 4 ms for a 512-state one of 32, whatever the number of families
// beside it. A cluster of eight CTAs therefore walks a tile of up to four
// families with one category, each CTA holding an eighth of the states of every
// vector; a parent gathers its child's whole vector through distributed shared
// memory. One cluster barrier per node. Many tiles run side by side and keep
// the pipe busy, and the four families share the matrix loads.
//
// k_term_tiles lists the tiles: a warp takes 32 families of a bin and, where
// some are flagged, the flagged ones of every category, four at a time, in any
// order (every tile writes its own terms).
//
// Measured (conversion, planning and recompute of a call; 32-family tiles of
// k_prune64, planned by one block, before): 10,000 families of 24 taxa, 96
// states, a few terms flagged 2.67 -> 0.15 ms; 20,000 of 48 taxa, 64 states, 64
// candidates with the eight rates of alpha = 0.5, small categories of 264 families
// flagged in each 34.3 -> 22.3 (6.0 with alpha from 0.5 to 1.13, where fewer terms
// are); nothing flagged 0.021 -> 0.020.
#include "common.cuh"

#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace cafe {
namespace {

constexpr int CL = 8;        // CTAs of a cluster
constexpr int NT = 128;
constexpr int G = 4;         // families of a tile (a warp each in the reductions)

__global__ void __launch_bounds__(256) k_term_tiles(TermTileArgs a) {
    if (*a.any_flag == 0) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    int64_t c = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);   // chunk of 32 families
    for (int b = 0; b < a.n_bins; ++b) {
        const int64_t chunks = (a.bin_count[b] + 31) / 32;
        for (; c < chunks; c += warps) {
            const int64_t i = 32 * c + lane;
            const int64_t first = a.bin_first[b] + 32 * c;
            const int64_t fam = i < a.bin_count[b] ? a.perm[first + lane] : -1;
            const bool flagged = fam >= 0 && a.flags[fam] != 0;
            const unsigned any = __ballot_sync(0xffffffffu, flagged);
            if (!any) continue;
            if (lane == 0) atomicAdd(&a.out_counts[0], __popc(any));
            for (int q = 0; q < a.n_cats; ++q) {
                const int k = a.cats[q];
                unsigned m = __ballot_sync(0xffffffffu, flagged && a.term_flags[(size_t)fam * a.K + k] != 0);
                if (!m || lane != 0) continue;
                int at = atomicAdd(&a.out_counts[1], (__popc(m) + G - 1) / G);
                while (m) {
                    TermTile t;
                    t.first = (int32_t)first;
                    t.mask = 0;
                    for (int g = 0; g < G && m; ++g) {
                        t.mask |= m & (0u - m);
                        m &= m - 1;
                    }
                    t.k = k;
                    t.W = a.bin_width[b];
                    a.tiles[at++] = t;
                }
            }
        }
        c -= chunks;
    }
}

__device__ __forceinline__ double warp_max(double x) {
    // values >= 0: the order of the bits
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, b, o);
        b = y > b ? y : b;
    }
    return __longlong_as_double((long long)b);
}

// The power of two the vector with these maxima is scaled by (frexp's exponent).
__device__ __forceinline__ int scale_of(const double* m) {
    unsigned long long b = 0;      // values >= 0: the order of the bits
    for (int r = 0; r < CL; ++r) {
        const unsigned long long y = (unsigned long long)__double_as_longlong(m[r]);
        b = y > b ? y : b;
    }
    const double x = __longlong_as_double((long long)b);
    int e = 0;
    if (x > 0.0 && isfinite(x)) frexp(x, &e);
    return e;
}

// scalbn(x, -e), by the exponent field where it stays within the normal range.
__device__ __forceinline__ double scaled_down(double x, int e) {
    const int hi = __double2hiint(x), ne = (hi >> 20) - e;
    if (hi >= 0x00100000 && ne > 0 && ne < 2047) return __hiloint2double(hi - e * 0x100000, __double2loint(x));
    return x == 0.0 ? x : scalbn(x, -e);
}

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(NT) k_terms64(TermArgs a) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int64_t fam[G];
    __shared__ int e_sh[G];
    __shared__ double root_v[G][CL];      // (of the cluster's first CTA)
    __shared__ int root_nz[G][CL];
    cg::cluster_group cluster = cg::this_cluster();
    const TreePlan& P = a.plan;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)cluster.block_rank();
    const int wmax = a.W / CL;
    double* part = sm;                                           // [n_slots][G][wmax] this CTA's states
    double* full = part + (size_t)P.n_slots * G * wmax;         // [G][W] a child's vector
    double* maxs = full + (size_t)G * a.W;                      // [n_slots][G][CL] largest value of each CTA's states
    int* exps = reinterpret_cast<int*>(maxs + (size_t)P.n_slots * G * CL);  // [n_slots][G] the children's exponents
    const int n_tiles = *a.n_tiles;
    if ((int)blockIdx.x / CL >= n_tiles) return;
    cluster.sync();      // the other CTAs run: their shared memory may be written
    for (int t = blockIdx.x / CL; t < n_tiles; t += gridDim.x / CL) {
        const TermTile tile = a.tiles[t];
        const int cnt = __popc(tile.mask), k = tile.k, W = tile.W, S = W - 1, w = W / CL, s0 = rank * w;
        if (tid < cnt) fam[tid] = a.perm[tile.first + __fns(tile.mask, 0, tid + 1)];
        __syncthreads();
        const double* const* mats = a.mats + (size_t)k * P.n_nodes;
        for (int ii = 0; ii < P.n_internal; ++ii) {
            const int vs = P.slot[P.internal[ii]];
            double* dst = part + (size_t)vs * G * wmax;
            if (tid < G) exps[vs * G + tid] = 0;
            for (int ci = P.cstart[ii]; ci < P.cstart[ii + 1]; ++ci) {
                const int ch = P.child[ci];
                const bool first = ci == P.cstart[ii];
                const double* __restrict__ M = mats[ch];
                const int lc = P.leaf_col[ch];
                if (lc >= 0) {
                    for (int idx = tid; idx < cnt * w; idx += NT) {
                        const int g = idx / w, sl = idx % w;
                        const int n = a.counts[(size_t)fam[g] * P.n_leaves + lc];
                        const double* Mr = M + (size_t)(s0 + sl) * a.ld_mat;
                        double val = 0.0;
                        if (a.err) {
                            const double* pr = a.err + (size_t)(n < a.err_rows ? n : a.err_rows - 1) * a.err_ndev;
                            const int off = n - (a.err_ndev - 1) / 2;
                            for (int d = 0; d < a.err_ndev; ++d) {
                                const int c = off + d;
                                if (c < 0 || c > S) continue;
                                val = fma(Mr[c], pr[d], val);
                            }
                        } else if (n >= 0 && n <= S) {
                            val = Mr[n];
                        }
                        double* o = dst + (size_t)g * wmax + sl;
                        *o = first ? val : *o * val;
                    }
                } else {
                    const int cs = P.slot[ch];
                    if (tid < cnt) {
                        const int e = scale_of(maxs + ((size_t)cs * G + tid) * CL);
                        e_sh[tid] = e;
                        exps[vs * G + tid] += exps[cs * G + tid] + e;
                    }
                    __syncthreads();
                    for (int idx = tid; idx < cnt * W; idx += NT) {
                        const int g = idx / W, j = idx % W, e = e_sh[g];
                        const double* src = cluster.map_shared_rank(part + ((size_t)cs * G + g) * wmax, j / w);
                        const double x = src[j % w];
                        full[(size_t)g * a.W + j] = scaled_down(x, e);
                    }
                    __syncthreads();
                    // four chains per state, over j = 0, 1, 2, 3 (mod 4): a warp takes
                    // eight states of one family (a warp issues an FP64 instruction
                    // every 64 clocks, so the families go side by side)
                    const int m = lane & 3;
                    for (int it = warp; it < (w + 7) / 8 * cnt; it += NT / 32) {
                        const int g = it % cnt, sl = it / cnt * 8 + (lane >> 2);
                        const double* Mr = M + (size_t)(s0 + min(sl, w - 1)) * a.ld_mat + m;
                        const double* L = full + (size_t)g * a.W + m;
                        double v = 0.0;
                        for (int j0 = 0; j0 < W; j0 += 32) {
                            double mv[8];
#pragma unroll
                            for (int h = 0; h < 8; ++h) mv[h] = __ldg(Mr + j0 + 4 * h);
#pragma unroll
                            for (int h = 0; h < 8; ++h) v = fma(mv[h], L[j0 + 4 * h], v);
                        }
                        v += __shfl_xor_sync(0xffffffffu, v, 1);
                        v += __shfl_xor_sync(0xffffffffu, v, 2);
                        if (m == 0 && sl < w) {
                            double* o = dst + (size_t)g * wmax + sl;
                            *o = first ? v : *o * v;
                        }
                    }
                }
                __syncthreads();
            }
            // the root's rows are the root sizes 1..S
            const int lo = ii == P.n_internal - 1 && rank == 0 ? 1 : 0;
            if (warp < cnt) {
                double mx = 0.0;      // (values >= 0: the order of the bits)
                for (int sl = lo + lane; sl < w; sl += 32) {
                    const double x = dst[(size_t)warp * wmax + sl];
                    mx = __double_as_longlong(x) > __double_as_longlong(mx) ? x : mx;
                }
                mx = warp_max(mx);
                if (lane < CL) cluster.map_shared_rank(maxs + ((size_t)vs * G + warp) * CL, lane)[rank] = mx;
            }
            cluster.sync();
        }
        // ---- root weighting (K4): a warp per family, then the first CTA ----
        const int rs = P.slot[P.root];
        if (warp < cnt) {
            const int e = scale_of(maxs + ((size_t)rs * G + warp) * CL);
            const int Rf = a.fam_R ? min(a.fam_R[fam[warp]], S) : S;
            double best = a.model == 0 ? -INFINITY : 0.0;
            int nz = 0;
            for (int sl = lane; sl < w; sl += 32) {
                const int j = s0 + sl - 1;        // root size j + 1
                if (j < 0 || j >= Rf) continue;
                double x = part[((size_t)rs * G + warp) * wmax + sl];
                x = scaled_down(x, e);
                const double eq = j < a.n_prior ? a.prior[j] : 0.0;
                const double v = a.model == 0 ? log(x) + log(eq) : x * eq;
                best = v > best ? v : best;
                nz |= x != 0.0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double y = __shfl_xor_sync(0xffffffffu, best, o);
                best = y > best ? y : best;
            }
            nz = __any_sync(0xffffffffu, nz);
            if (lane == 0) {
                e_sh[warp] = e;      // (the maxima may be the next tile's after the barrier)
                cluster.map_shared_rank(&root_v[0][0], 0)[warp * CL + rank] = best;
                cluster.map_shared_rank(&root_nz[0][0], 0)[warp * CL + rank] = nz;
            }
        }
        cluster.sync();
        if (rank == 0 && tid < cnt) {
            double b = root_v[tid][0];
            int nz = 0;
            for (int r = 0; r < CL; ++r) {
                b = root_v[tid][r] > b ? root_v[tid][r] : b;
                nz |= root_nz[tid][r];
            }
            const double E = (double)(exps[rs * G + tid] + e_sh[tid]) * 0.69314718055994530942;
            double o;
            if (a.model == 0) o = b + E;
            else o = nz ? log(b * a.cat_probs[k]) + E : NAN;      // (an all-zero root vector: the family fails)
            a.out[(size_t)fam[tid] * a.K + k] = o;
        }
        __syncthreads();
    }
}

constexpr int kMaxDynSmem = 200 * 1024;

// (trees without polytomies, so at most a dozen slots: 42 KB at 512 states)
size_t terms_smem(int W, int n_slots) {
    return G * (((size_t)n_slots * (W / CL) + (size_t)W + (size_t)n_slots * CL) * sizeof(double) +
                       (size_t)n_slots * sizeof(int));
}

}  // namespace

// Tiles at most: every term of every listed category flagged.
int64_t term_tiles_max(int64_t F, int n_bins, int n_cats) { return (F / 32 + n_bins) * (int64_t)(32 / G) * n_cats; }

cudaError_t terms64_init() {
    return cudaFuncSetAttribute(k_terms64, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
}

cudaError_t launch_term_tiles(const TermTileArgs& a, int sm_count, cudaStream_t s) {
    int64_t chunks = 0;
    for (int b = 0; b < a.n_bins; ++b) chunks += (a.bin_count[b] + 31) / 32;
    if (chunks <= 0 || a.n_cats <= 0) return cudaSuccess;
    k_term_tiles<<<(unsigned)std::min<int64_t>((chunks + 7) / 8, 2 * sm_count), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_terms64(const TermArgs& a, int sm_count, cudaStream_t s) {
    const size_t smem = terms_smem(a.W, a.plan.n_slots);
    // (the walks wait on barriers: with four CTAs per SM the 264 families above
    // take 35 ms, with 12 24, with 20, more than fit at a time, 22)
    const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(20, (size_t)kMaxDynSmem / smem));
    k_terms64<<<std::max(1, sm_count * per_sm / CL) * CL, NT, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace cafe
