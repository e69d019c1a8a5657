// K1: birth-death transition matrices in FP64, one CTA per (lambda, t) key.
//
// Replaces matrix_cache::precalculate_matrices (src/matrix_cache.cpp:113-163)
// over birthdeath_rate_with_log_alpha (src/probability.cpp:104-148), which
// evaluates P(s -> c) = sum_j C(s,j) C(s+c-j-1, s-1) a^(s+c-2j) (1-2a)^j with
// one exp and one pow per term: O(S^3) terms per matrix. On GB300 FP64 is
// the scarcest pipe, so this kernel uses an O(S^2) scheme instead:
//
//  * Row s is the coefficient sequence of G(z)^s, G(z) = (a + b z)/(1 - a z)
//    with a = lt/(1+lt), b = 1 - 2a (the one-lineage law P(1->0) = a,
//    P(1->c) = (1-a)^2 a^(c-1)). From (a + b z)(1 - a z) G_s' = s(1-a)^2 G_s:
//        g_{c+1} = [ ((s-c) b + a^2 (s+c)) g_c + a b (c-1) g_{c-1} ] / (a (c+1))
//    For c < s both coefficients are >= 0, so the forward recurrence only
//    adds non-negative terms and is stable; it starts at g_0 = a^s.
//  * The upper triangle follows from c P(s->c) = s P(c->s) (the two
//    binomial sums differ term by term by the factor s/c): the chain of row
//    s also writes P(c->s) = (c/s) P(s->c) into rows c < s.
//  * Both kinds of store leave each warp as contiguous row segments (the
//    lower triangle through a shared-memory staging tile).
//  * The running value is kept as mantissa * 2^E so rows whose left end
//    underflows FP64 (a^s < 1e-308) still reach their diagonal exactly.
//
// Row 0 is delta(c,0); a key whose 1 - 2a is not in (0, 1) has zero rows
// s >= 1 (the_probability_of_going_from_parent_fam_size_to_c,
// src/probability.cpp:150-167, and the saturation rule of
// matrix_cache.cpp:139-154). Entries are clamped to <= 1 as in
// probability.cpp:147.
#include "common.cuh"

#include <algorithm>

namespace cafe {
namespace {

constexpr double kLn2Hi = 6.93147180369123816490e-01;  // Cody-Waite split of ln 2
constexpr double kLn2Lo = 1.90821492927058770002e-10;

// min(m 2^e, 1), m >= 0, e <= 0: the exponent is added as an integer; only
// results just below the normal range take an FP64 instruction (one rounding,
// as scalbn's). x: the result's exponent field.
__device__ __noinline__ double small_value(double m, int e, int x) {
    if (e == 0) return m;
    const int hi = __double2hiint(m);
    if (hi < 0x00100000) return scalbn(m, e);      // itself below the normal range
    return __hiloint2double((hi & 0xfffff) | (x + 64) << 20, __double2loint(m)) * 0x1p-64;
}
__device__ __forceinline__ double out_value(double m, int e) {
    const int hi = __double2hiint(m), x = (hi >> 20) + e;
    if (x < 1 && x >= -63) return small_value(m, e, x);
    const double v = __hiloint2double(hi + e * 0x100000, __double2loint(m));
    return x >= 1023 ? 1.0 : x < 1 ? 0.0 : v;
}

// Per-matrix coefficient tables in shared memory (k = 0..W):
//   p1[c] = (q + alpha) / (c + 1), p2[c] = c (alpha - q) / (c + 1)
//     so that ((s - c) q + alpha (s + c)) / (c + 1) = s p1[c] + p2[c]
//   bb[c] = (1 - 2 alpha) (c - 1) / (c + 1)
struct Coeffs {
    const double* p1;
    const double* p2;
    const double* bb;
};

// (a call, so that no step issues the product predicated off, which would take
// the FP64 pipe all the same)
__device__ __noinline__ double down600(double x) { return x * 0x1p-600; }

// One row chain: the coefficients g_c of row s, c = 0..s, as a running
// mantissa m times 2^E; cs = c / s for the mirrored entry of row c. The
// coefficients of the step to come, a and t = bb[c] g_{c-1}, are formed a step
// ahead, so that a step waits for one FMA.
struct RowChain {
    int s, E;
    double m, a, t, sd, inv_s, cs;

    __device__ void init(int s_, double la, const Coeffs& k) {
        s = s_;
        const double L0 = (double)s * la;  // log(a^s)
        E = 0;
        if (L0 > -700.0) {
            m = exp(L0);
        } else {
            E = (int)floor(L0 * 1.4426950408889634) + 1;
            m = exp((L0 - (double)E * kLn2Hi) - (double)E * kLn2Lo);
        }
        sd = (double)s;
        a = fma(sd, k.p1[0], k.p2[0]);
        t = k.bb[0] * 0.0;
        inv_s = 1.0 / sd;
        cs = 0.0;
    }
    __device__ __forceinline__ double value() const { return out_value(m, E); }
    // g_c -> g_{c+1}: two FMAs and a product per step
    __device__ __forceinline__ void advance(int c, const Coeffs& k) {
        const double nx = fma(a, m, t);
        a = fma(sd, k.p1[c + 1], k.p2[c + 1]);
        t = k.bb[c + 1] * m;
        cs += inv_s;
        m = nx;
        if (__double2hiint(nx) >= 0x65800000) {   // g >= 2^601
            m = down600(m);
            t = down600(t);
            E += 600;
        }
    }
};

constexpr int kStageCols = 8;    // steps of a warp's staging tile
constexpr int kStagePitch = 33;  // padded row pitch (doubles) of the staging tile

// `parts` CTAs of T threads per matrix, each with an equal share of its row
// pairs, so a side-512 build spreads over the SMs in small CTAs. A lane owns
// the rows W - 1 - p and 1 + p, one straight after the other: W + 2 entries
// whatever p is, so no lane of a warp waits for another (what bounds the kernel
// is the FP64 pipe: five instructions a step; with few matrices the latency of
// the chain). The second row's start is prepared with the first one's. Each
// step writes the mirror P(c->s) = (c/s) P(s->c) into row c < s (in the lanes'
// first rows contiguous across the warp), and puts P(s->c) into a tile of
// eight steps in shared memory, which leaves as contiguous row segments. Row 0 is
// delta(c, 0).
//
// Measured (a warp's longest row of each half in turn and scalbn for every
// entry of a row whose left end underflows, before; build and staging): 204
// matrices of side 768 1.77 -> 0.73 ms, 40,448 of side 64 1.99 -> 1.09, 148 of
// side 96 0.075 -> 0.050, 18 of side 171 0.114 -> 0.071. A warp alone on its
// quarter of an SM issues an FP64 instruction every 64 clocks, which is what the
// small builds take.
__global__ void __launch_bounds__(128) k_matrix_build(const MatrixJob* __restrict__ jobs, int parts) {
    extern __shared__ double sh[];
    const int part = blockIdx.x % parts;
    const MatrixJob J = jobs[blockIdx.x / parts];
    const int W = J.size;
    double* p1 = sh;                   // coefficient tables (Coeffs), k = 0..W
    double* p2 = p1 + (W + 1);
    double* bb = p2 + (W + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* stage = bb + (W + 1) + (size_t)warp * kStageCols * kStagePitch;
    double* M = J.dst;
    const double lt = J.lambda * J.t;
    const double alpha = lt / (1 + lt);
    const double coeff = 1 - 2 * alpha;
    const bool live = (coeff > 0 && coeff != 1);
    const double q = live ? coeff / alpha : 0.0;
    if (part == 0)
        for (int c = threadIdx.x; c < W; c += blockDim.x) M[c] = (c == 0) ? 1.0 : 0.0;
    if (!live) {
        const size_t stride = (size_t)parts * blockDim.x;
        for (size_t i = (size_t)W + (size_t)part * blockDim.x + threadIdx.x; i < (size_t)W * W; i += stride) M[i] = 0.0;
        return;
    }
    for (int k = threadIdx.x; k <= W; k += blockDim.x) {
        const double ik = 1.0 / (double)(k + 1);
        p1[k] = (q + alpha) * ik;
        p2[k] = (double)k * (alpha - q) * ik;
        bb[k] = coeff * ((double)(k - 1) * ik);
    }
    const Coeffs cf{p1, p2, bb};
    __syncthreads();
    const double la = log(alpha);
    const int npairs = W / 2;   // rows 1..W-1 in pairs (the middle row once when W is even)
    for (int p0 = part * blockDim.x + warp * 32; p0 < npairs; p0 += parts * blockDim.x) {
        const int p = p0 + lane;
        RowChain ch, second;
        ch.s = second.s = -1;      // (no row)
        if (p < npairs) {
            ch.init(W - 1 - p, la, cf);
            if (1 + p != ch.s) second.init(1 + p, la, cf);
        }
        int c = 0;
        for (int t0 = 0; t0 < W + 2; t0 += kStageCols) {
            // no lane reaches its row's end in this tile, and all are in their first
            // rows, or all in their second: no checks (column 0's mirror is row 0's
            // own zero), and the tile's rows lie a fixed stride apart
            const bool act = p < npairs, one = ch.s == W - 1 - p;
            const bool run = c + kStageCols <= ch.s;
            const bool firsts = __all_sync(0xffffffffu, !act || (run && one));
            if (firsts || __all_sync(0xffffffffu, !act || (run && !one))) {
                double* up = M + (size_t)c * W + ch.s;
                const Coeffs kc{p1 + c, p2 + c, bb + c};
#pragma unroll
                for (int cc = 0; cc < kStageCols; ++cc) {
                    const double v = ch.value();
                    stage[cc * kStagePitch + lane] = v;
                    if (act) *up = ch.cs * v;
                    up += W;
                    ch.advance(cc, kc);
                }
                c += kStageCols;
                __syncwarp();
                const int r = lane / kStageCols, col = lane % kStageCols;
                const double* st = stage + col * kStagePitch + r;
                const int64_t stride = firsts ? -(int64_t)W : (int64_t)W + 1;
                double* o = firsts ? M + (int64_t)(W - 1 - p0 - r) * W + t0 + col
                                   : M + (int64_t)(1 + p0 + r) * W + t0 - W + p0 + r + col;
                const int rows = npairs - p0 - r;
#pragma unroll
                for (int i = 0; i < 32; i += 32 / kStageCols) {
                    if (i < rows) *o = st[i];
                    o += 32 / kStageCols * stride;
                }
                __syncwarp();
                continue;
            }
#pragma unroll 4
            for (int cc = 0; cc < kStageCols; ++cc) {
                if (c <= ch.s) {
                    const double v = ch.value();
                    stage[cc * kStagePitch + lane] = v;
                    if (c < ch.s) {
                        if (c > 0) M[(size_t)c * W + ch.s] = ch.cs * v;      // (c / s < 1, v <= 1)
                        ch.advance(c, cf);
                        ++c;
                    } else {      // (the diagonal)
                        ch = second;
                        second.s = -1;
                        c = 0;
                    }
                }
            }
            __syncwarp();
            // the tile's rows, several per warp instruction
            for (int idx = lane; idx < 32 * kStageCols; idx += 32) {
                const int r = idx / kStageCols, t = t0 + idx % kStageCols;
                const int pr = p0 + r, s1 = W - 1 - pr, s2 = 1 + pr, c2 = t - s1 - 1;
                const double v = stage[(idx % kStageCols) * kStagePitch + r];
                if (pr >= npairs) continue;
                if (t <= s1) M[(size_t)s1 * W + t] = v;
                else if (s2 != s1 && c2 <= s2) M[(size_t)s2 * W + c2] = v;
            }
            __syncwarp();
        }
    }
}

}  // namespace

cudaError_t launch_matrix_build(const MatrixJob* d_jobs, int n_jobs, int max_size, int sm_count, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    // one thread per row pair, in whole warps, and as many CTAs per matrix as
    // its pairs need: one warp each while that gives at most four per SM, then
    // two, which share the tables
    const int pairs = max_size / 2;
    const int warps = std::max(1, (pairs + 31) / 32);
    const int threads = warps == 1 || (int64_t)n_jobs * warps <= 4 * sm_count ? 32 : 64;
    const int parts = std::max(1, (pairs + threads - 1) / threads);
    size_t smem = sizeof(double) * (3 * (size_t)(max_size + 1) + (size_t)(threads / 32) * kStageCols * kStagePitch);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_matrix_build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k_matrix_build<<<n_jobs * parts, threads, smem, s>>>(d_jobs, parts);
    return cudaGetLastError();
}

}  // namespace cafe
