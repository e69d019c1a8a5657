// Around the tensor-core pruning (k_pat_tc.cu): conversion of the FP64
// matrices into its operands, and the plan of the FP64 recompute of the
// category terms it could not represent or whose range bound is too large.
#include "common.cuh"
#include "tc_ptx.cuh"

#include <math.h>

#include <algorithm>

namespace cafe {
namespace {

// FP64 matrix -> TF32 hi/lo operands (row-major, pitch Wm) and the FP32
// transpose tr[c][s] = M[s][c] (a leaf factor, column c of M, as one row).
// With an error model the transpose's row c is already the leaf factor of
// an observed count c: sum_d w_d(c) M[s][c - h + d] over the model's 2h + 1
// deviations, in deviation order, as FP32 products and sums (the walk then
// reads one row per leaf, whatever the model's width). A block converts a
// band of 32 rows of one matrix, 32 columns (plus h on either side) at a
// time through a shared-memory tile, so the row-major and the transposed
// stores both write whole 128-byte lines. Wm is a multiple of 32.
__global__ void __launch_bounds__(256) k_convert_tc(const ConvertJob* __restrict__ jobs, TcBuffers b) {
    constexpr int TW = 32 + 2 * kMaxErrHalf;
    __shared__ float tile[32][TW + 1];
    __shared__ float wsh[32][2 * kMaxErrHalf + 1];   // the band's rows' deviation weights (0: skipped)
    const int Wm = b.Wm;
    const int bands = Wm / 32;
    const ConvertJob J = jobs[blockIdx.x / bands];
    const int s0 = (int)(blockIdx.x % bands) * 32;
    const size_t base = (size_t)J.mat * Wm * Wm;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int h = b.err ? (b.err_ndev - 1) / 2 : 0;
    // only what the walk reads: hi/lo for internal children's branches, the
    // transpose for leaves' (block-uniform)
    const bool want_hl = (J.what & 1) != 0, want_tr = (J.what & 2) != 0;
    // the deviations' columns either side of a 32-column step (within
    // 0 .. Wm - 1): lane tx < 2h loads column c0 + hoff into tile column hcol
    const bool halo = want_tr && tx < 2 * h;
    const int hoff = tx < h ? tx - h : 32 + (tx - h);
    const int hcol = tx < h ? tx : 32 + tx;
    for (int c0 = 0; c0 < Wm; c0 += 32) {
        // the thread's four rows (ty + 8 i) of this step, and their halo
        // entries, are loaded before any store (the stores might alias the
        // source as far as the compiler knows), so the loads overlap
        const int c = c0 + tx, cc = c0 + hoff;
        float x[4], xh[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = (float)J.src[(size_t)(s0 + ty + 8 * i) * J.ld + c];
        if (halo) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                xh[i] = (cc >= 0 && cc < Wm) ? (float)J.src[(size_t)(s0 + ty + 8 * i) * J.ld + cc] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + 8 * i, s = s0 + r;
            if (want_hl) {
                const float hi = tc::round_tf32(x[i]);
                b.hi[base + (size_t)s * Wm + c] = hi;
                b.lo[base + (size_t)s * Wm + c] = tc::round_tf32(x[i] - hi);
            }
            if (!want_tr) continue;
            tile[r][h + tx] = x[i];
            if (halo) tile[r][hcol] = xh[i];
        }
        if (!want_tr) continue;
        if (b.err)
            for (int q = threadIdx.x; q < 32 * b.err_ndev; q += blockDim.x) {
                const int r = q / b.err_ndev, d = q % b.err_ndev, c = c0 + r, col = c - h + d;
                const double w = b.err[(size_t)(c < b.err_rows ? c : b.err_rows - 1) * b.err_ndev + d];
                wsh[r][d] = (col >= 0 && col < Wm && w > 0) ? (float)w : 0.0f;
            }
        __syncthreads();
        for (int r = ty; r < 32; r += 8) {
            const int c = c0 + r;      // the count (row of tr); tx: the state s0 + tx
            float v;
            if (!b.err) {
                v = tile[tx][r];
            } else {
                // a skipped deviation has weight 0 here: fmaf(0, x, v) = v
                v = 0.0f;
                for (int d = 0; d < b.err_ndev; ++d) v = fmaf(wsh[r][d], tile[tx][r + d], v);
            }
            b.tr[base + (size_t)c * Wm + s0 + tx] = v;
        }
        __syncthreads();
    }
}

// One thread per (family, candidate): the category terms' range-error
// bounds weighted by their shares of the family likelihood; a family over
// tau |lnL| is flagged for the FP64 recompute. Terms that are not finite
// (a dead or failed category) carry no weight; a family none of whose
// terms is finite is left to the finish. The FP64 exponentials are what it
// costs, and an FP32 estimate settles nearly every family: 20,000 families x
// 512 terms 0.53 -> 0.061 ms.
__global__ void __launch_bounds__(256) k_range_flags(RangeFlagArgs a) {
    const int n_cand = a.K / a.KC;
    const int64_t n = a.F * n_cand;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = i / n_cand;
        const int b = (int)(i % n_cand);
        const double* c = a.cat + (size_t)f * a.K + (size_t)b * a.KC;
        const float* e = a.err + (size_t)f * a.K + (size_t)b * a.KC;
        uint8_t* tf = a.term_flags + (size_t)f * a.K + (size_t)b * a.KC;
        {
            // FP32 first: the terms' shares within 1e-3, the log likelihood within
            // 1e-3; most families are under budget by far
            float mf = -INFINITY, wf = 0.0f, wef = 0.0f;
            bool open = false;
            for (int k = 0; k < a.KC; ++k) {
                const float x = (float)c[k];
                if (isfinite(x)) mf = fmaxf(mf, x);
                open |= tf[k] != 0;
            }
            if (!(mf > -INFINITY)) continue;
            for (int k = 0; k < a.KC; ++k) {
                const float x = (float)c[k];
                if (!isfinite(x)) continue;
                const float s = __expf(x - mf);
                wf += s;
                wef += s * e[k];
            }
            if (!open && wef <= 0.98f * (float)a.tau * (fabsf(mf + __logf(wf)) - 0.01f) * wf) continue;
        }
        double m = -INFINITY;
        for (int k = 0; k < a.KC; ++k)
            if (isfinite(c[k])) m = fmax(m, c[k]);
        if (!(m > -INFINITY)) continue;
        double w = 0.0, we = 0.0;
        for (int k = 0; k < a.KC; ++k) {
            if (!isfinite(c[k])) continue;
            const double x = exp(c[k] - m);
            w += x;
            we += x * (double)e[k];
        }
        // a term the walk left to the FP64 pass carries no weight here, so the
        // others' shares are unknown: every term of the candidate is recomputed
        bool walk = false;
        for (int k = 0; k < a.KC; ++k) walk |= tf[k] != 0;
        if (walk) {
            for (int k = 0; k < a.KC; ++k) tf[k] = 1;
            continue;      // (the family is flagged already)
        }
        if (!(we != 0.0)) continue;      // no range loss in any term (or a candidate that was not pruned)
        const double lnl = m + log(w);
        const double bound = we / w;
        const double lim = a.tau * fabs(lnl);
        if (!(bound <= lim)) {
            // recompute the terms whose share of the bound is over lim / (2 KC):
            // the others' shares add up to at most lim / 2
            const double each = lim * w / (2.0 * a.KC);
            for (int k = 0; k < a.KC; ++k) {
                const bool fin = isfinite(c[k]);
                const double share = fin ? exp(c[k] - m) * (double)e[k] : 0.0;
                if (!(share <= each) || !(lim > 0.0)) tf[k] = 1;
            }
            atomicOr(&a.flags[f], 2);
            atomicOr(a.any_flag, 1);
        }
    }
}

}  // namespace

cudaError_t launch_range_flags(const RangeFlagArgs& a, cudaStream_t s) {
    const int64_t n = a.F * (a.K / a.KC);
    if (n <= 0) return cudaSuccess;
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, 4096);
    k_range_flags<<<blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_convert_tc(const ConvertJob* d_jobs, int n_jobs, TcBuffers b, cudaStream_t s) {
    if (n_jobs <= 0) return cudaSuccess;
    if (b.Wm % 32) return cudaErrorInvalidValue;
    k_convert_tc<<<(unsigned)(n_jobs * (b.Wm / 32)), 256, 0, s>>>(d_jobs, b);
    return cudaGetLastError();
}

}  // namespace cafe
