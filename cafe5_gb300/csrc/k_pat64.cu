// K3/K4 (FP64) over distinct rows: Felsenstein pruning where every node
// contracts each distinct count pattern of its subtree once.
//
// The arithmetic is that of k_prune64, and so are the bits: a row's vector
// is the product of its children's factors in descendant order, rescaled by
// a power of two in the scaled modes; its factor for the parent is
//   F[s] = sum_j M[s][j] L[j]
// as four FMA chains over j = 0, 1, 2, 3 (mod 4) in ascending j, combined as
// (s0 + s1) + (s2 + s3). Replaces the same reference functions
// (compute_node_probability, src/probability.cpp:175-234; matrix::multiply,
// src/matrix_cache.cpp:32-58; the root reductions of src/base_model.cpp:77-95
// and src/gamma_core.cpp:143-165).
//
// What bounds it is the FP64 pipe (two FMAs a clock and SM), so the kernel
// does fewer FMAs, and everything else is arranged around that:
//  * rows are the distinct patterns (k_patterns.cu), 4.4 times fewer than
//    families x nodes on 10,000 families of 24 taxa;
//  * a warp leaves out a 32-column chunk of the sum when every term in it is
//    below 2^-55 of every partial sum it would join (exponents of the
//    chunk's largest M and |L| against the smallest partial sum): each of
//    those FMAs would return its addend unchanged, so the bits stay. L
//    falls off geometrically past the observed counts, and with the
//    reference's global bound (171 states for counts up to 35) most of the
//    upper columns go;
//  * states are cut to the vector's length, not to whole 64-row passes.
// Measured (kernel time, 32-family tiles walking every node before): 10,000
// families of 24 taxa, K = 4, 171 states 59.3 -> 6.5 ms; 50,000 of 32 taxa in
// bins of 32 to 768 15.0 -> 4.5 ms; 2,777 of 17 taxa, K = 5, error model
// 1.85 -> 0.57 ms; 1,000 of 12 taxa, 171 states 1.08 (a cluster per family)
// -> 0.26 ms, where the nine dependent levels are the bound.
// A unit is 8 rows x s_run tiles of 16 states: the pipe is so
// narrow that 8 x 16 x 171 FMAs keep one SM busy for 6 us, so small units
// spread a tree level over the SMs, and many CTAs per SM keep the pipe fed
// while others load. One producer warp per CTA takes the next unit, waits for
// the factors it reads and forms its rows' vectors in shared memory while
// the four compute warps are still at the unit before; those read the matrix
// through L1 and never meet a barrier inside a unit.
//
// One persistent launch walks all combined categories. A unit is (node, row
// tile, state tiles) of one combination; units come from a counter, ordered
// by the node's height, so a unit's children were handed out before it to
// CTAs that are running: it waits (bounded) for their count of finished
// units, and the wait always ends (a CTA's own units come in order too).
// `group` combinations are interleaved unit by unit, which keeps every SM
// busy across a tree level's end; factor tables exist for n_slots
// combinations at a time, and a combination's first writer waits for the
// root of the one whose table it takes over.
#include "common.cuh"
#include "flog2.cuh"

#include <math.h>

#include <algorithm>

namespace cafe {
namespace {

constexpr int NT = 128;      // compute threads
constexpr int NTHR = NT + 32;   // and the producer warp
constexpr int TP = kPat64Rows;     // rows of a unit
constexpr int TS = kPat64States;   // states of a tile: four per compute warp
constexpr int KC = 32;       // columns of a chunk of the sums
constexpr int kFewRows = 4;
constexpr int BJ = 16;       // columns whose matrix entries are loaded together
constexpr int kMaxChunks = 256;
constexpr int kWaitPolls = 1 << 26;
constexpr int kDescSh = 512; // nodes whose first units are kept in shared memory

// Named barriers: a vector buffer filled, a buffer free again, the compute
// warps among themselves.
enum { kFull = 1, kEmpty = 3, kCompute = 5 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    __threadfence_block();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// High word of a value >= 0, with 0 only for an exact zero.
__device__ __forceinline__ int hi_key(double x) {
    const int h = __double2hiint(x);
    return h ? h : (__double2loint(x) ? 1 : 0);
}
// The same of |x|, for vectors: they can hold negative values (a search over an
// error model's epsilon may try a negative one). A negative partial sum needs none:
// its word is below every exponent's, and then no chunk is left out.
__device__ __forceinline__ int hi_key_abs(double x) {
    const int h = __double2hiint(x) & 0x7fffffff;
    return h ? h : (__double2loint(x) ? 1 : 0);
}
// 0 < p <= infinity, on the integer pipe.
__device__ __forceinline__ bool has_log(double p) {
    return (unsigned long long)(__double_as_longlong(p) - 1) < 0x7ff0000000000000ull;
}

// One thread: wait until *p has reached n.
__device__ __forceinline__ bool wait_count(const int32_t* p, int n, const int32_t* status) {
    for (int i = 0; i < kWaitPolls; ++i) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= n) return true;
        if ((i & 15) == 15 && *(const volatile int32_t*)status) return false;
        __nanosleep(100);
    }
    return false;
}

// A node's children as a unit reads them: factor rows of the combination's
// table. The first two are set up once (in shared memory), further ones
// (polytomies) at every use.
struct ChildTab {
    const double* base;
    int64_t pitch;        // from one row to the next
    int32_t rows;
    const int32_t* expo;  // exponents of the rows, null for a leaf
};
struct NodeSrcs {
    ChildTab c[2];
    int nch;
};

__device__ __forceinline__ ChildTab child_tab(const Pat64Args& a, const Pat64Node& nd, const double* tab,
                                              const int32_t* expo, int c) {
    const Pat64Node& cn = a.nodes[a.cdesc[nd.child0 + c]];
    return ChildTab{tab + cn.tab, cn.pitch, cn.rows, cn.nch ? expo + cn.erow0 : nullptr};
}

// (a leaf's last row stands for every larger count)
__device__ __forceinline__ const double* child_row(const ChildTab& t, int idx) {
    return t.base + (int64_t)min(idx, t.rows - 1) * t.pitch;
}

struct RowSrc {
    const double *s0, *s1;
    const int32_t* idx;   // the row's child indices
};

__device__ __forceinline__ RowSrc row_src(const Pat64Args& a, const Pat64Node& nd, const NodeSrcs& ns, int row, int i0,
                                          int i1) {
    RowSrc r;
    r.idx = a.child + nd.cidx + (int64_t)row * ns.nch;
    r.s0 = child_row(ns.c[0], i0);
    r.s1 = ns.nch > 1 ? child_row(ns.c[1], i1) : r.s0;
    return r;
}

// Product over the children at state j, in descendant order.
__device__ __forceinline__ double product(const Pat64Args& a, const Pat64Node& nd, const NodeSrcs& ns, const RowSrc& r,
                                          const double* tab, const int32_t* expo, int j) {
    double v = __ldcg(r.s0 + j);
    if (ns.nch > 1) v *= __ldcg(r.s1 + j);
    for (int c = 2; c < ns.nch; ++c) v *= __ldcg(child_row(child_tab(a, nd, tab, expo, c), __ldg(r.idx + c)) + j);
    return v;
}

// Sum of the internal children's power-of-two exponents of a row.
__device__ __forceinline__ int child_exp(const Pat64Args& a, const Pat64Node& nd, const NodeSrcs& ns, const RowSrc& r,
                                         const double* tab, const int32_t* expo) {
    int E = 0;
    for (int c = 0; c < ns.nch; ++c) {
        const ChildTab t = c < 2 ? ns.c[c] : child_tab(a, nd, tab, expo, c);
        if (t.expo) E += __ldcg(t.expo + __ldg(r.idx + c));
    }
    return E;
}

// A leaf's factor rows: row n is column n of the branch's matrix (the count
// n's one-hot vector through it), or the error model's weighted sum of the
// columns n - h .. n + h within the states. One element per thread and step,
// neighbouring threads on neighbouring states' rows.
__device__ void leaf_rows(const Pat64Args& a, const Pat64Node& nd, const double* M, double* tab, int p0, int tid, int nt) {
    const int np = min(kPat64Rows, nd.n_list - p0);
    for (int e = tid; e < np * nd.s_cnt; e += nt) {
        const int s = e / np;                        // (neighbouring counts share sectors)
        const int n = min(__ldg(a.leaf_counts + nd.cidx + p0 + e % np), nd.rows - 1);
        const double* Mr = M + (size_t)s * a.ld_mat;
        double val = 0.0;
        if (a.err) {
            const double* pr = a.err + (size_t)(n < a.err_rows ? n : a.err_rows - 1) * a.err_ndev;
            const int off = n - (a.err_ndev - 1) / 2;
            for (int d = 0; d < a.err_ndev; ++d) {
                const int c = off + d;
                if (c < 0 || c > nd.S) continue;
                val = fma(__ldg(Mr + c), pr[d], val);
            }
        } else if (n <= nd.S) {
            val = __ldg(Mr + n);
        }
        tab[nd.tab + (int64_t)n * nd.pitch + s] = val;
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

// The power of two a row with maximum m is scaled by (frexp's exponent).
__device__ __forceinline__ int scale_exp(double m) {
    int e = 0;
    if (m > 0.0 && isfinite(m)) frexp(m, &e);
    return e;
}

// Root weighting of one family per warp (K4): the arithmetic of k_prune64.
__device__ void root_family(const Pat64Args& a, const Pat64Node& nd, const NodeSrcs& ns, const double* tab,
                            const int32_t* expo, int k, int row, double* x, int lane) {
    const int32_t* ci = a.child + nd.cidx + (int64_t)row * ns.nch;
    const RowSrc rs = row_src(a, nd, ns, row, __ldg(ci), ns.nch > 1 ? __ldg(ci + 1) : 0);
    const int R = nd.R;
    if (a.root_out) {
        double* o = a.root_out + (size_t)a.perm[nd.perm0 + row] * R;
#pragma unroll 4
        for (int j = lane; j < R; j += 32) o[j] = product(a, nd, ns, rs, tab, expo, 1 + j);
        return;
    }
    int E = a.scaled ? child_exp(a, nd, ns, rs, tab, expo) : 0;
    double mx = 0.0;
#pragma unroll 4
    for (int j = lane; j < R; j += 32) {
        const double v = product(a, nd, ns, rs, tab, expo, 1 + j);
        x[j] = v;
        mx = v > mx ? v : mx;
    }
    if (a.scaled) {
        const int e = scale_exp(warp_max(mx));
        E += e;
        if (e != 0)
            for (int j = lane; j < R; j += 32) x[j] = scalbn(x[j], -e);
    }
    const int64_t f = a.perm[nd.perm0 + row];
    const int Rf = a.fam_R ? min(a.fam_R[f], R) : R;
    double o;
    if (a.model == 0) {
        // max_j log x + log eq, evaluated only where the FP32 logarithms (each
        // within 1.3e-4) come within 2^-6 of the best (of priors above 0: others,
        // NaN among them, have no logarithm)
        float top = -INFINITY;
        for (int j = lane; j < Rf; j += 32)
            if (j < a.n_prior && has_log(a.prior[j])) top = fmaxf(top, flog2(x[j]) + flog2(a.prior[j]));
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, q));
        double best = -INFINITY;
        if (top > -INFINITY)
            for (int j = lane; j < Rf; j += 32)
                if (j < a.n_prior && has_log(a.prior[j]) && flog2(x[j]) + flog2(a.prior[j]) >= top - 0.015625f) {
                    const double v = log(x[j]) + log(a.prior[j]);
                    best = v > best ? v : best;
                }
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, best, q);
            best = y > best ? y : best;
        }
        o = best + (double)E * 0.69314718055994530942;
    } else {
        double m = 0.0;
        int nz = 0;
        for (int j = lane; j < Rf; j += 32) {
            const double eq = j < a.n_prior ? a.prior[j] : 0.0;
            const double v = x[j] * eq;
            m = v > m ? v : m;
            nz |= x[j] != 0.0;
        }
        m = warp_max(m);
        nz = __any_sync(0xffffffffu, nz);
        const double cat = m * a.cat_probs[k];
        if (!nz) o = a.scaled ? NAN : -1.0;   // all-zero root vector: family fails
        else if (a.scaled) o = log(cat) + (double)E * 0.69314718055994530942;
        else o = cat;
    }
    if (lane == 0) a.out[(size_t)f * a.K + k] = o;
    __syncwarp();
}

// What the producer hands to the compute warps.
struct Unit {
    Pat64Node nd;
    NodeSrcs src;
    double* tab;
    int32_t* expo;
    int32_t* ctab;        // max-product: argmax table, laid out like tab
    const double* M;      // the branch's matrix (null at the root)
    int q, k, di, p0, t0, t1, is_root, stop;
};

// Max-product: where a buffer keeps the FP32 logarithms of its vectors.
struct LogRows {
    float* lu;     // [TP][pitch] log2 u, -inf past the states
    int pitch;     // rows 16 bytes apart modulo 128
    float* cm;     // [TP][chunks] its largest value in each chunk
    int* peak;     // [TP] where it is largest
};
__host__ __device__ inline size_t log_rows_doubles(int nchunk) {
    return ((size_t)TP * (nchunk * KC + 4) + (size_t)TP * nchunk + TP + 1) / 2;
}
__device__ __forceinline__ LogRows log_rows(double* Ls, int nchunk) {
    LogRows r;
    r.lu = reinterpret_cast<float*>(Ls + (size_t)TP * (nchunk * KC + 2));
    r.pitch = nchunk * KC + 4;
    r.cm = r.lu + (size_t)TP * r.pitch;
    r.peak = reinterpret_cast<int*>(r.cm + (size_t)TP * nchunk);
    return r;
}

// The unit's eight vectors, four lanes per row: 32 states (16 loads a lane)
// in flight before the first product.
// Max-product: also their log2 in FP32, its largest value per chunk, and where
// it is largest.
template <bool MX>
__device__ __forceinline__ void fill_rows(const Pat64Args& a, const Unit& u, double* Ls, int* lmax, int idx_pack,
                                          int lane) {
    const Pat64Node& nd = u.nd;
    const int S = nd.S, nchunk = S / KC + 1, lp = nchunk * KC + 2;
    const int l = lane & 3, r = lane >> 2;
    const int row = min(u.p0 + r, nd.rows - 1);      // rows past the last repeat it
    const int i0 = __shfl_sync(0xffffffffu, idx_pack, 2 * r), i1 = __shfl_sync(0xffffffffu, idx_pack, 2 * r + 1);
    const RowSrc rs = row_src(a, nd, u.src, row, i0, i1);
    const bool two = u.src.nch == 2;
    double* L = Ls + (size_t)r * lp;
    double mx = 0.0;
    const LogRows lr = log_rows(Ls, nchunk);
    float top = -INFINITY;
    int top_j = 0;
    for (int ck = 0; ck < nchunk; ++ck) {
        const int j0 = ck * KC + l;
        double x[8];
        if (two) {
            double y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int j = j0 + 4 * i;
                x[i] = j <= S ? __ldcg(rs.s0 + j) : 0.0;
                y[i] = j <= S ? __ldcg(rs.s1 + j) : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] *= y[i];
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int j = j0 + 4 * i;
                x[i] = j <= S ? product(a, nd, u.src, rs, u.tab, u.expo, j) : 0.0;
            }
        }
        if (MX) {
            float cm = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int j = j0 + 4 * i;
                L[j] = x[i];
                const float lu = j <= S ? flog2(x[i]) : -INFINITY;
                lr.lu[r * lr.pitch + j] = lu;
                cm = fmaxf(cm, lu);
                if (lu > top) {
                    top = lu;
                    top_j = j;
                }
            }
            cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, 1));
            cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, 2));
            if (l == 0) lr.cm[r * nchunk + ck] = cm;
            continue;
        }
        int m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            L[j0 + 4 * i] = x[i];
            mx = x[i] > mx ? x[i] : mx;
            m = max(m, hi_key_abs(x[i]));
        }
        if (!a.scaled) {
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) lmax[ck] = m;
        }
    }
    if (MX) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, top, o);
            const int j = __shfl_xor_sync(0xffffffffu, top_j, o);
            if (t > top) {
                top = t;
                top_j = j;
            }
        }
        if (l == 0) lr.peak[r] = top_j;
        return;
    }
    if (!a.scaled) return;
    unsigned long long mb = (unsigned long long)__double_as_longlong(mx);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, mb, o);
        mb = y > mb ? y : mb;
    }
    const int e = scale_exp(__longlong_as_double((long long)mb));
    for (int ck = 0; ck < nchunk; ++ck) {
        int m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            double x = L[ck * KC + l + 4 * i];
            if (e != 0) {
                x = scalbn(x, -e);
                L[ck * KC + l + 4 * i] = x;
            }
            m = max(m, hi_key_abs(x));
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) lmax[ck] = m;
    }
    // the rows' exponents, once per row (the unit of its first states)
    if (u.t0 == 0 && l == 0 && u.p0 + r < nd.rows) u.expo[nd.erow0 + row] = e + child_exp(a, nd, u.src, rs, u.tab, u.expo);
}

// The vectors of a unit of at most four rows (few_rows reads no others): the
// warp's lanes along the states, four chunks in flight.
__device__ __forceinline__ void fill_few(const Pat64Args& a, const Unit& u, double* Ls, int* lmax, int idx_pack, int np,
                                         int lane) {
    const Pat64Node& nd = u.nd;
    const int S = nd.S, nchunk = S / KC + 1, lp = nchunk * KC + 2;
    const bool two = u.src.nch == 2;
    for (int r = 0; r < np; ++r) {
        const int i0 = __shfl_sync(0xffffffffu, idx_pack, 2 * r), i1 = __shfl_sync(0xffffffffu, idx_pack, 2 * r + 1);
        const RowSrc rs = row_src(a, nd, u.src, u.p0 + r, i0, i1);
        double* L = Ls + (size_t)r * lp;
        double mx = 0.0;
        for (int c0 = 0; c0 < nchunk; c0 += 4) {
            double x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = (c0 + i) * KC + lane;
                x[i] = j > S ? 0.0 : two ? __ldcg(rs.s0 + j) : product(a, nd, u.src, rs, u.tab, u.expo, j);
                y[i] = two && j <= S ? __ldcg(rs.s1 + j) : 1.0;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (c0 + i >= nchunk) break;
                if (two) x[i] *= y[i];
                L[(c0 + i) * KC + lane] = x[i];
                mx = x[i] > mx ? x[i] : mx;
                if (!a.scaled) {
                    const int m = __reduce_max_sync(0xffffffffu, hi_key_abs(x[i]));
                    if (lane == 0) lmax[c0 + i] = r ? max(lmax[c0 + i], m) : m;
                }
            }
        }
        if (!a.scaled) continue;
        const int e = scale_exp(warp_max(mx));
        for (int ck = 0; ck < nchunk; ++ck) {
            double x = L[ck * KC + lane];
            if (e != 0) {
                x = scalbn(x, -e);
                L[ck * KC + lane] = x;
            }
            const int m = __reduce_max_sync(0xffffffffu, hi_key_abs(x));
            if (lane == 0) lmax[ck] = r ? max(lmax[ck], m) : m;
        }
        // the row's exponent, once per row (the unit of its first states)
        if (u.t0 == 0 && lane == 0)
            u.expo[nd.erow0 + u.p0 + r] = e + child_exp(a, nd, u.src, rs, u.tab, u.expo);
    }
}

// The producer warp: units into the buffers in turn.
template <bool MX>
__device__ void produce(const Pat64Args& a, Unit* units, double* Ls, size_t buf_doubles, int (*lmax)[kMaxChunks],
                        const int* unit0_sh, int lane) {
    const long long total = (long long)a.units * a.n_active;
    // the next unit is taken while the current one is prepared (its turn comes
    // after a smaller one's, so the order that ends every wait still holds)
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(a.next, 1ull);
    for (int it = 0;; ++it) {
        const int b = it % a.n_bufs;
        if (it >= a.n_bufs) bar_sync(kEmpty + b, NTHR);
        Unit& u = units[b];
        const long long idx = (long long)__shfl_sync(0xffffffffu, next, 0);
        bool ok = idx < total;
        if (ok) {
            if (lane == 0) next = atomicAdd(a.next, 1ull);
            // (combination, unit): `group` combinations interleaved
            const long long per = (long long)a.units * a.group;
            const int g0 = (int)(idx / per) * a.group;
            const int gn = min(a.group, a.n_active - g0);
            const int rem = (int)(idx % per);
            const int ui = rem / gn, q = g0 + rem % gn;
            int lo = 0, hi = a.n_desc - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((mid < kDescSh ? unit0_sh[mid] : a.nodes[mid].unit0) <= ui) lo = mid;
                else hi = mid - 1;
            }
            const Pat64Node& nd = a.nodes[lo];
            const int v = nd.node, nch = nd.nch, ul = ui - nd.unit0;
            const bool is_root = nd.root == lo;
            const int k = a.active[q], slot = q % a.n_slots;
            double* tab = a.table + (size_t)slot * a.slot_doubles;
            int32_t* expo = a.expo + (size_t)slot * a.slot_rows;
            const double* const* mats = a.mats + (size_t)k * a.plan.n_nodes;
            const int p0 = is_root ? ul * kPat64RootRows : (ul / nd.s_tiles) * TP;
            if (lane == 0) {
                u.nd = nd;
                u.tab = tab;
                u.expo = expo;
                u.ctab = MX ? a.ctab + (size_t)slot * a.slot_doubles : nullptr;
                u.M = is_root ? nullptr : mats[v];
                u.q = q;
                u.k = k;
                u.di = lo;
                u.p0 = p0;
                u.t0 = nch == 0 || is_root ? 0 : (ul % nd.s_tiles) * a.s_run;
                u.t1 = nch == 0 || is_root ? 0 : min(u.t0 + a.s_run, (nd.s_cnt + TS - 1) / TS);
                u.is_root = is_root;
                u.stop = 0;
                u.src.nch = nch;
            }
            if (lane < 2 && lane < nch) u.src.c[lane] = child_tab(a, nd, tab, expo, lane);
            // the rows' first two child indices (lane 2 r + c)
            int pack = 0;
            if (!is_root && lane < 2 * TP && (lane & 1) < nch)
                pack = __ldg(a.child + nd.cidx + (int64_t)min(p0 + (lane >> 1), nd.rows - 1) * nch + (lane & 1));
            // lane c waits for child c, lane 31 for the table's last user
            bool w = true;
            if (lane == 0) w = *(volatile int32_t*)a.status == 0;
            for (int c = lane; w && c < nch; c += 31) {
                if (lane == 31) break;
                const int d = a.cdesc[nd.child0 + c];
                w = wait_count(a.done + (size_t)q * a.n_desc + d, a.nodes[d].n_units, a.status);
            }
            if (lane == 31 && q >= a.n_slots)
                w = wait_count(a.done + (size_t)(q - a.n_slots) * a.n_desc + nd.root, a.nodes[nd.root].n_units, a.status);
            ok = __all_sync(0xffffffffu, w);
            __syncwarp();      // what one lane waited for, every lane reads
            if (ok && !is_root && nch > 0) {
                const int np = min(TP, nd.rows - p0);
                if (!MX && np <= kFewRows) fill_few(a, u, Ls + b * buf_doubles, lmax[b], pack, np, lane);
                else fill_rows<MX>(a, u, Ls + b * buf_doubles, lmax[b], pack, lane);
            }
            if (!ok && lane == 0) atomicExch(a.status, 1);
        }
        if (!ok && lane == 0) u.stop = 1;
        __syncwarp();
        bar_arrive(kFull + b, NTHR);
        if (!ok) return;
    }
}

// A unit of at most four rows: lanes are 8 states x the sums' 4 chains, so an
// FMA serves 32 products whatever the row count (with a row per lane group a
// lone row would cost as much as eight: the widest bins hold a handful of
// families). The same chains, leave-out test and sum as below.
__device__ __forceinline__ void few_rows(const Pat64Args& a, const Unit& u, const double* Lb, int lp, int np, int nchunk,
                                         const int* lmax, int warp, int lane) {
    const int S = u.nd.S, s_cnt = u.nd.s_cnt;
    const int m = lane & 3, st = lane >> 2;
    for (int sb = u.t0 * TS + warp * 8; sb < min(u.t1 * TS, s_cnt); sb += 8 * (NT / 32)) {
        const int s = sb + st;
        const double* Mr = u.M + (size_t)min(s, s_cnt - 1) * a.ld_mat;
        double nx[KC / 4];
        auto fetch = [&](int ck) {
#pragma unroll
            for (int h = 0; h < KC / 4; ++h) {
                const int j = ck * KC + 4 * h + m;
                nx[h] = j <= S ? __ldg(Mr + j) : 0.0;
            }
        };
        fetch(0);
        double acc[kFewRows];
#pragma unroll
        for (int r = 0; r < kFewRows; ++r) acc[r] = 0.0;
        for (int ck = 0; ck < nchunk; ++ck) {
            double mv[KC / 4];
            int mk = 0;
#pragma unroll
            for (int h = 0; h < KC / 4; ++h) {
                mv[h] = nx[h];
                mk = max(mk, hi_key(mv[h]));
            }
            bool skip = false;
            if (ck > 0) {
                const int lk = lmax[ck];
                int am = 0x7fffffff;
#pragma unroll
                for (int r = 0; r < kFewRows; ++r)
                    if (r < np) am = min(am, __double2hiint(acc[r]));
                const int ea = am >> 20;
                skip = mk == 0 || lk == 0 || (ea > 0 && (mk >> 20) + (lk >> 20) + 2 <= ea + 968);
                skip = __all_sync(0xffffffffu, skip);
            }
            if (ck + 1 < nchunk) fetch(ck + 1);
            if (skip) continue;
            const double* Lt = Lb + ck * KC + m;
#pragma unroll
            for (int r = 0; r < kFewRows; ++r) {
                if (r >= np) continue;
#pragma unroll
                for (int h = 0; h < KC / 4; ++h) acc[r] = fma(mv[h], Lt[(size_t)r * lp + 4 * h], acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < kFewRows; ++r) {
            if (r >= np) continue;
            double v = acc[r];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (m == 0 && s < s_cnt) u.tab[u.nd.tab + (int64_t)(u.p0 + r) * u.nd.pitch + s] = v;
        }
    }
}

// ---- max-product (Pupko joint reconstruction): L[i] = max_j u[j] M[i][j] and
// the first j attaining it, in FP64, as k_pupko defines it: the products are
// ranked by FP32 logarithms (each p = log2 u + log2 M within 5e-4 of exact),
// and only those within kDelta of the best are formed in FP64.
//
// A chunk of 32 columns is left out for a (row, state) whose best so far is
// kDelta above the sum of the chunk's largest log2 u and largest log2 M: no
// product in it can be the maximum. "Best so far" starts from the products at
// the row's peak and at j = i, so most rows look at one or two chunks.
//
// What bounds it is the producer warp, which forms a vector's logarithms; a
// unit therefore runs over up to 16 state tiles. Measured (device time of the
// whole call, every family walking every node in 32-family tiles before):
// 10,000 families of 24 taxa, K = 4, 85 states 20.0 -> 1.2 ms.
constexpr float kDelta = 0.00390625f;   // 2^-8, in log2 units

// FP64 over the candidate child states, ascending: one queued (row, state) per
// lane.
__device__ __forceinline__ void slow_rows(const Pat64Args& a, const Unit& u, const double* Lb, const LogRows& lr,
                                          const float* lm, const float* cmM, int nchunk, const int* pair,
                                          const float* best, int count, int lane) {
    if (lane < count) {
        const int S = u.nd.S, lp = nchunk * KC + 2;
        const int r = pair[lane] & 7, i = pair[lane] >> 3;
        const float b1 = best[lane], thr = b1 - kDelta;
        const bool all = !(b1 > -INFINITY);
        const double* Mi = u.M + (size_t)i * a.ld_mat;
        double mx = -1.0;
        int arg = 0;
        for (int c = 0; c < nchunk; ++c) {
            if (!all && !(lr.cm[r * nchunk + c] + cmM[(size_t)i * nchunk + c] >= thr)) continue;
            for (int j = c * KC; j < min(c * KC + KC, S + 1); ++j) {
                if (!all && !(lr.lu[r * lr.pitch + j] + lm[(size_t)i * a.lm_pitch + j] >= thr)) continue;
                const double val = Lb[(size_t)r * lp + j] * __ldg(Mi + j);
                if (val > mx) {
                    mx = val;
                    arg = j;
                }
            }
        }
        const int64_t at = u.nd.tab + (int64_t)(u.p0 + r) * u.nd.pitch + i;
        u.tab[at] = mx;
        u.ctab[at] = arg;
    }
    __syncwarp();
}

__device__ __forceinline__ void max_rows(const Pat64Args& a, const Unit& u, double* Lb, int* pair, float* slow, int warp,
                                         int lane) {
    const int pl = lane & 7, sl = lane >> 3;
    const int S = u.nd.S, s_cnt = u.nd.s_cnt, nchunk = S / KC + 1, lp = nchunk * KC + 2;
    const int np = min(TP, u.nd.rows - u.p0);
    const LogRows lr = log_rows(Lb, nchunk);
    const float* lm = a.lmats[(size_t)u.k * a.plan.n_nodes + u.nd.node];     // [S + 1][lm_pitch]
    const float* cmM = lm + (size_t)(S + 1) * a.lm_pitch;                    // [S + 1][nchunk]
    const float* LU = lr.lu + pl * lr.pitch;
    int queued = 0;
    for (int t = u.t0; t < u.t1; ++t) {
        if (t * TS + warp * 4 >= s_cnt) break;
        const int i = t * TS + warp * 4 + sl;
        const int ic = min(i, s_cnt - 1);
        const float* LM = lm + (size_t)ic * a.lm_pitch;
        const float* CM = cmM + (size_t)ic * nchunk;
        const int pk = lr.peak[pl];
        // a product's logarithm: no more than the best one's
        const float floor_b = fmaxf(LU[pk] + __ldg(LM + pk), LU[ic] + __ldg(LM + ic));
        float b1 = -INFINITY, b2 = -INFINITY;
        int j1 = 0;
        for (int c = 0; c < nchunk; ++c) {
            const bool look = lr.cm[pl * nchunk + c] + __ldg(CM + c) >= fmaxf(floor_b, b1) - kDelta;
            if (!__any_sync(0xffffffffu, look)) continue;
#pragma unroll
            for (int q = 0; q < KC; q += 4) {
                const float4 x = *reinterpret_cast<const float4*>(LU + c * KC + q);
                const float4 y = __ldg(reinterpret_cast<const float4*>(LM + c * KC + q));
                const float p[4] = {x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    j1 = p[h] > b1 ? c * KC + q + h : j1;
                    b2 = fmaxf(b2, fminf(b1, p[h]));
                    b1 = fmaxf(b1, p[h]);
                }
            }
        }
        const bool valid = pl < np && i < s_cnt;
        const bool zero = !(b1 >= -1075.0f - kDelta);      // every product rounds to 0
        const bool near_sub = b1 < -1022.0f + kDelta;
        const bool fast = !near_sub && b2 < b1 - kDelta;   // only j1 can reach the FP64 maximum
        if (valid && (zero || fast)) {
            const int64_t at = u.nd.tab + (int64_t)(u.p0 + pl) * u.nd.pitch + i;
            u.tab[at] = fast ? Lb[(size_t)pl * lp + j1] * __ldg(u.M + (size_t)i * a.ld_mat + j1) : 0.0;
            u.ctab[at] = fast ? j1 : 0;
        }
        // the rest (near-ties, rows near the subnormal range) are queued and
        // scanned a warp at a time
        const bool slow_it = valid && !zero && !fast;
        const unsigned m = __ballot_sync(0xffffffffu, slow_it);
        if (slow_it) {
            const int at = queued + __popc(m & ((1u << lane) - 1u));
            pair[at] = pl | i << 3;
            slow[at] = near_sub ? -INFINITY : b1;
        }
        queued += __popc(m);
        __syncwarp();
        if (queued >= 32) {
            slow_rows(a, u, Lb, lr, lm, cmM, nchunk, pair + queued - 32, slow + queued - 32, 32, lane);
            queued -= 32;
        }
    }
    slow_rows(a, u, Lb, lr, lm, cmM, nchunk, pair, slow, queued, lane);
}

// reconstruct_root_node (src/gene_family_reconstructor.cpp:47-78): the first
// root size j in 1..R with the largest prod_children L[j] * prior(j).
__device__ __forceinline__ void root_argmax(const Pat64Args& a, const Pat64Node& nd, const NodeSrcs& ns, const double* tab,
                                            const int32_t* expo, int k, int row, int lane) {
    const int32_t* ci = a.child + nd.cidx + (int64_t)row * ns.nch;
    const RowSrc rs = row_src(a, nd, ns, row, __ldg(ci), ns.nch > 1 ? __ldg(ci + 1) : 0);
    double best = -1.0;
    int arg = 0;
#pragma unroll 2
    for (int j = 1 + lane; j <= nd.R; j += 32) {
        const double val = product(a, nd, ns, rs, tab, expo, j) * (j < a.n_prior ? a.prior[j] : 0.0);
        if (val > best) {
            best = val;
            arg = j;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double b = __shfl_xor_sync(0xffffffffu, best, o);
        const int j = __shfl_xor_sync(0xffffffffu, arg, o);
        if (b > best || (b == best && j < arg)) {
            best = b;
            arg = j;
        }
    }
    if (lane == 0) {
        const int64_t f = a.perm[nd.perm0 + row];
        a.root_max[(size_t)k * a.F + f] = best;
        a.root_arg[(size_t)k * a.F + f] = arg;
        if (!(best > 0.0)) atomicAdd(a.n_failed, 1);
    }
}

// Four compute warps along the states of a tile: lanes 8 rows x 4 states.
template <bool MX>
__global__ void __launch_bounds__(NTHR, 6) k_pat64(const Pat64Args a) {
    extern __shared__ __align__(16) double Ls[];   // [n_bufs][buf_doubles]: [TP][lp] (root units: [4][R])
    __shared__ int lmax[2][kMaxChunks];            // largest L of each chunk (hi_key)
    __shared__ Unit units[2];
    __shared__ int unit0_sh[kDescSh];              // first units of the nodes
    __shared__ int slow_pair[MX ? NT / 32 : 1][64];
    __shared__ float slow_best[MX ? NT / 32 : 1][64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < min(a.n_desc, kDescSh); i += NTHR) unit0_sh[i] = a.nodes[i].unit0;
    __syncthreads();
    if (warp == NT / 32) {
        produce<MX>(a, units, Ls, a.buf_doubles, lmax, unit0_sh, lane);
        return;
    }
    const int pl = lane & 7, sl = lane >> 3;
    for (int it = 0;; ++it) {
        const int buf = it % a.n_bufs;
        bar_sync(kFull + buf, NTHR);
        const Unit& u = units[buf];
        if (u.stop) return;
        const double* Lb = Ls + buf * a.buf_doubles;
        if (MX && u.is_root) {
            for (int i = warp; i < kPat64RootRows && u.p0 + i < u.nd.rows; i += NT / 32)
                root_argmax(a, u.nd, u.src, u.tab, u.expo, u.k, u.p0 + i, lane);
        } else if (MX && u.src.nch > 0) {
            max_rows(a, u, Ls + buf * a.buf_doubles, slow_pair[warp], slow_best[warp], warp, lane);
        } else if (u.is_root) {
            double* x = Ls + buf * a.buf_doubles + (size_t)warp * u.nd.R;
            for (int i = warp; i < kPat64RootRows && u.p0 + i < u.nd.rows; i += NT / 32)
                root_family(a, u.nd, u.src, u.tab, u.expo, u.k, u.p0 + i, x, lane);
        } else if (u.src.nch == 0) {
            leaf_rows(a, u.nd, u.M, u.tab, u.p0, tid, NT);
        } else {
            const int S = u.nd.S, s_cnt = u.nd.s_cnt;
            const int nchunk = S / KC + 1, lp = nchunk * KC + 2;
            const int np = min(TP, u.nd.rows - u.p0);
            const double* L = Lb + (size_t)pl * lp;
            if (np <= kFewRows) few_rows(a, u, Lb, lp, np, nchunk, lmax[buf], warp, lane);
            else for (int t = u.t0; t < u.t1; ++t) {
                if (t * TS + warp * 4 >= s_cnt) break;       // no states for this warp
                // this thread's row of the matrix (past the last: the last again)
                const int sr = t * TS + warp * 4 + sl;
                const double* Mr = u.M + (size_t)min(sr, s_cnt - 1) * a.ld_mat;
                // its share of the row's chunk ck: the values the leave-out test
                // looks at, loaded a chunk ahead, which also brings the chunk into L1
                double pf[KC / 8];
                auto fetch = [&](int ck) {
#pragma unroll
                    for (int h = 0; h < KC / 8; ++h) {
                        const int j = ck * KC + pl + 8 * h;
                        pf[h] = j <= S ? __ldg(Mr + j) : 0.0;
                    }
                };
                fetch(0);
                double acc[4] = {0.0, 0.0, 0.0, 0.0};
                for (int ck = 0; ck < nchunk; ++ck) {
                    bool skip = false;
                    if (ck > 0) {
                        // leave the chunk out when no term in it can change a partial sum
                        const int lk = lmax[buf][ck];
                        int mk = 0;
#pragma unroll
                        for (int h = 0; h < KC / 8; ++h) mk = max(mk, hi_key(pf[h]));
#pragma unroll
                        for (int o = 1; o < 8; o <<= 1) mk = max(mk, __shfl_xor_sync(0xffffffffu, mk, o));
                        const int am = min(min(__double2hiint(acc[0]), __double2hiint(acc[1])),
                                           min(__double2hiint(acc[2]), __double2hiint(acc[3])));
                        const int ea = am >> 20;
                        skip = mk == 0 || lk == 0 || (ea > 0 && (mk >> 20) + (lk >> 20) + 2 <= ea + 968);
                        skip = __all_sync(0xffffffffu, skip);
                    }
                    if (ck + 1 < nchunk) fetch(ck + 1);
                    if (skip) continue;
                    const int jn = min(KC, S + 1 - ck * KC);
                    const double* Lt = L + ck * KC;
                    const double* Mt = Mr + ck * KC;
                    // whole blocks of 16 columns: the matrix loads ahead of the sums
                    int jj = 0;
                    for (; jj + BJ <= jn; jj += BJ) {
                        double m[BJ];
#pragma unroll
                        for (int h = 0; h < BJ; ++h) m[h] = __ldg(Mt + jj + h);
#pragma unroll
                        for (int h = 0; h < BJ; h += 2) {
                            const double2 l = *reinterpret_cast<const double2*>(Lt + jj + h);
                            acc[h & 3] = fma(m[h], l.x, acc[h & 3]);
                            acc[(h & 3) + 1] = fma(m[h + 1], l.y, acc[(h & 3) + 1]);
                        }
                    }
                    for (; jj < jn; jj += 4) {
                        double m[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) m[h] = jj + h < jn ? __ldg(Mt + jj + h) : 0.0;
#pragma unroll
                        for (int h = 0; h < 4; ++h) acc[h] = fma(m[h], Lt[jj + h], acc[h]);
                    }
                }
                if (pl < np && sr < s_cnt)
                    u.tab[u.nd.tab + (int64_t)(u.p0 + pl) * u.nd.pitch + sr] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
            }
        }
        // every compute thread's rows are written before the unit counts as
        // finished; the producer's exponents came before its barrier
        bar_sync(kCompute, NT);
        if (tid == 0) {
            __threadfence();
            atomicAdd(a.done + (size_t)u.q * a.n_desc + u.di, 1);
        }
        __syncwarp();
        bar_arrive(kEmpty + buf, NTHR);
    }
}

// Doubles of one vector buffer.
size_t buf_doubles(int lp, int max_R, bool max_product) {
    const size_t n = max_product ? (size_t)TP * lp + log_rows_doubles((lp - 2) / KC)
                                 : std::max<size_t>((size_t)TP * lp, (size_t)(NT / 32) * max_R);
    return (n + 1) & ~(size_t)1;
}

constexpr int kMaxDynSmem = 200 * 1024;

}  // namespace

// Vector buffers of a launch (two where they fit), 0 when not even one does.
int pat64_bufs(int lp, int max_R, bool max_product) {
    if (lp - 2 > kMaxChunks * KC) return 0;
    const size_t n = buf_doubles(lp, max_R, max_product) * sizeof(double);
    return 2 * n <= (size_t)kMaxDynSmem ? 2 : n <= (size_t)kMaxDynSmem ? 1 : 0;
}
int64_t pat64_buf_doubles(int lp, int max_R, bool max_product) { return (int64_t)buf_doubles(lp, max_R, max_product); }

cudaError_t pat64_init() {
    const cudaError_t e = cudaFuncSetAttribute(k_pat64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_pat64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
}

int pat64_ctas_per_sm(size_t smem, bool max_product) {
    int n = 0;
    const cudaError_t e = max_product ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_pat64<true>, NTHR, smem)
                                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_pat64<false>, NTHR, smem);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return std::max(1, n);
}

cudaError_t launch_pat64(const Pat64Args& a, int n_ctas, cudaStream_t s) {
    if (a.units <= 0 || a.n_active <= 0) return cudaSuccess;
    const size_t smem = (size_t)a.n_bufs * a.buf_doubles * sizeof(double);
    if (a.ctab) k_pat64<true><<<n_ctas, NTHR, smem, s>>>(a);
    else k_pat64<false><<<n_ctas, NTHR, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace cafe
