// K3/K4 on the tensor cores over distinct rows: split-TF32 (TF32x3) pruning
// where every node contracts each distinct count pattern of its subtree
// (k_patterns.cu) once.
//
// Same algorithm and arithmetic as the FP64 kernels (inference_prune,
// src/core.cpp:134-145 -> compute_node_probability,
// src/probability.cpp:175-234 -> matrix::multiply, src/matrix_cache.cpp:32-58;
// root weighting src/gamma_core.cpp:143-165), in FP32 with integer exponents:
//
//  * A node's row is the product of its children's factor rows: a leaf's is a
//    row of the FP32 transposed matrix (with an error model: the weighted sum
//    of its columns, k_convert_tc), an internal child's a row of its factor
//    table. The row is brought back to [0.5, 1) by a power of two when its
//    maximum drifts below 2^-32; where the product underflows, the factors are
//    scaled apart before it, by the largest per-state sum of their binary
//    exponents (more than 2^250 apart: the family is left to FP64).
//  * Its factor for the parent is a GEMM D[row][s] = sum_j L[row][j] M[s][j]:
//    128 rows x W (or a share of at most 128 states) x W, operands split into
//    TF32 hi and lo parts, D = hi*hi + hi*lo + lo*hi per 8 columns
//    (tcgen05.mma kind::tf32, FP32 accumulators in TMEM). D goes through
//    shared memory into the node's factor table by TMA stores.
//  * At the root a family's two factors are weighted by the prior (root index
//    j = state j + 1) and the category term's natural log is written in FP64.
//  * FP32 range: every row carries an absolute error bound E (in its own
//    normalised units): a factor of an internal child is off by at most
//    E_child + 8 W 2^-126 (flushed matrix entries, flushed lo parts and
//    products; rows of M sum to <= 1), a leaf factor by a few 2^-126 where its
//    value is below 2^-100; the product's bound is u_A (f_B + u_B) + u_B f_A,
//    scaled like the product. At the root the bound of the best prior-weighted
//    row, relative to it, is written per (family, category); families whose
//    weighted bound exceeds tau |lnL| are recomputed in FP64 (k_range_flags).
//  * Without an error model every state-0 entry is exact (row 0 of every matrix
//    is delta(s, 0)), so a product that is zero everywhere at a node with a
//    saturated child is exactly zero: the row is dead and its families' terms
//    are log 0.
//
// What bounds it: the bytes of the factor rows between L2 and the SMs (about
// 1 KB per row of 64 states), not the tensor pipe. So rows are distinct
// patterns, a row is read once per parent row, and loads of many rows are in
// flight per thread. A walk of whole families up the tree (one tile per CTA,
// 19.5k clocks per tile and node) was bound by the latency of its node chain;
// here a unit's inputs are complete before it starts and units of different
// nodes and combinations fill the SMs.
//
// One persistent launch per S-bin. A unit is (node, 128 rows, state share) of
// one combination; units come from a counter, in segments of one tree level of
// a block of combinations, the blocks skewed by a level each: neighbouring
// segments are independent, and a unit's inputs were handed out a whole step
// earlier, to CTAs that are running, so every wait for them (bounded) ends.
// Factor tables exist for n_slots combinations at a time; a combination's
// units wait for the root of the one whose table they take over. The skew keeps
// levels + 1 blocks of tables alive; where memory has room for fewer, the blocks'
// segments follow one another unskewed, and one table is enough.
//
// Roles in a CTA: a scheduler warp (units, their inputs' completion, child
// indices), an issuer (TMA, MMA, completion) and 4 or 8 data warps (rows:
// copies, product, split; epilogue). All waits are bounded; on time-out the
// kernel records a status, drains its own copies and MMAs, frees TMEM and
// returns.
//
// Measured (each bin alone; families walked up the tree before): 16 x 4
// combinations of 10,000 families of 24 taxa, W = 64 1,490 -> 547 us, W = 32
// 645 -> 139, W = 96 399 -> 99; 64 x 8 of 20,000 families of 48 taxa 54 -> 9.7
// ms. W = 64 moves 0.91 GB of DRAM in its 547 us (25 % of a copy's rate), the
// tensor pipe is 8 % active; the rest is the latency of gathered rows.
#include "common.cuh"
#include "tc_ptx.cuh"

#include <math.h>

#include <algorithm>
#include <atomic>

namespace cafe {
namespace {

constexpr int TM = 128;      // rows per unit = MMA M = TMEM lanes
constexpr int KC = 32;       // columns per chunk: one 128-byte swizzle row
constexpr int kChunkA = TM * KC;         // floats of one A chunk (hi or lo)
constexpr int kPolls = 1 << 26;          // of a count in global memory
constexpr int kBarPolls = 1 << 20;       // of a barrier in shared memory
constexpr int kSegSh = 64;   // segments whose first units are kept in shared memory
constexpr int kNodeSh = 32;  // and nodes kept there
constexpr float kTiny = 0x1p-126f;       // smallest normal FP32 value
constexpr int32_t kSatBit = 1 << 30;     // of a matrix index: the key is saturated
enum { kFlag = 1, kDead = 2 };           // row flags

__device__ __forceinline__ int bexp(float y) {
    // binary exponent e with y = m 2^e, m in [0.5, 1); zero -> very negative
    const uint32_t b = __float_as_uint(y);
    const int be = (int)((b >> 23) & 0xFF);
    if (!(y > 0.0f)) return -100000;
    return be ? be - 126 : -149;
}
__device__ __forceinline__ float pow2f(int a) {
    a = a < -126 ? -126 : (a > 127 ? 127 : a);
    return __uint_as_float((uint32_t)(a + 127) << 23);
}

__device__ __align__(16) float g_one_row[512];      // the factor of an absent second child (1; pat_tc_init fills it)

constexpr int NB = 3;         // units in hand: one done with, one worked on, one prepared

// One unit, as the scheduler hands it to the issuer and the data warps.
struct Info {
    const float* tab[2];      // the children's factor rows
    const int4* meta[2];      // an internal child's row records; null: a leaf
    int pitch[2];
    int nch, np, is_root, sat, k, stop;
    int q, di, row_out, s_off, mat;      // combination, node, first table row, first state, matrix
    int4* meta_out;           // the unit's own row records
    int64_t item0;            // root: first item
    int idx[2][TM];           // child indices of the rows
};

// Record of a factor row: x = exponent << 2 | flags, y = error bound, and
// (bins of up to 64 states) z, w = the largest factor value of each 32 columns.

// What the scaling of a row's product and its error bound rest on.
struct RowStat {
    float maxp, fmx0, fmx1, fmn0, fmn1;
};

__device__ __forceinline__ float max4(const float4& a) { return fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)); }
__device__ __forceinline__ float min4(const float4& a) { return fminf(fminf(a.x, a.y), fminf(a.z, a.w)); }
__device__ __forceinline__ float maxprod4(const float4& a, const float4& b) {
    return fmaxf(fmaxf(a.x * b.x, a.y * b.y), fmaxf(a.z * b.z, a.w * b.w));
}
__device__ __forceinline__ float lane8_max(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float lane8_min(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ void stat_init(RowStat& t) {
    t.maxp = t.fmx0 = t.fmx1 = 0.0f;
    t.fmn0 = t.fmn1 = 1.0f;
}
__device__ __forceinline__ void stat_add4(RowStat& t, const float4& a, const float4& b) {
    t.maxp = fmaxf(t.maxp, maxprod4(a, b));
    t.fmx0 = fmaxf(t.fmx0, max4(a));
    t.fmx1 = fmaxf(t.fmx1, max4(b));
    t.fmn0 = fminf(t.fmn0, min4(a));
    t.fmn1 = fminf(t.fmn1, min4(b));
}
// A row's sources: its children's factor rows, and whether a leaf's count was
// outside the bin (FP64 recomputes such a family: any row serves).
struct Row {
    int n0, n1;
    int fl;
};
// What an internal child's record adds.
struct RowMeta {
    int E, fl;
    float er0, er1;       // error bounds of the factors (a leaf's: where it falls below 2^-100)
    float fm0, fm1;       // largest factor values of internal children (bins of up to 64 states)
};

// Whether a leaf's factor row of count n stands for the count exactly. With
// an error model, row n of the transposed matrix holds the weighted sum over
// columns 0 .. Wm - 1: the bin's own columns 0 .. S when the deviations stay
// within S; otherwise, or with no column of positive weight, FP64 recomputes.
__device__ __forceinline__ bool leaf_ok(const PatTcArgs& a, int n) {
    const int S = a.W - 1;
    if (!a.err) return n <= S;
    const int h = (a.err_ndev - 1) / 2;
    if (n > S - h) return false;
    const double* pr = a.err + (size_t)(n < a.err_rows ? n : a.err_rows - 1) * a.err_ndev;
    for (int d = max(0, h - n); d < a.err_ndev; ++d)
        if (__ldg(pr + d) > 0) return true;
    return false;
}

__device__ __forceinline__ Row make_row(const PatTcArgs& a, const Info& I, int r) {
    Row w{0, 0, 0};
    if (r >= I.np) return w;      // (a padding row: nothing reads what comes of it)
    w.n0 = I.idx[0][r];
    w.n1 = I.idx[1][r];
    if (!I.meta[0] && !leaf_ok(a, w.n0)) {
        w.fl = kFlag;
        w.n0 = 0;
    }
    if (!I.meta[1] && !leaf_ok(a, w.n1)) {
        w.fl = kFlag;
        w.n1 = 0;
    }
    return w;
}

// (issued with the first loads, decoded once the rows are done)
struct RawMeta {
    int4 q0, q1;
};
__device__ __forceinline__ RawMeta load_meta(const Info& I, int r, const Row& w) {
    RawMeta q{make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
    if (r >= I.np) return q;
    if (I.meta[0]) q.q0 = __ldcg(I.meta[0] + w.n0);
    if (I.nch > 1 && I.meta[1]) q.q1 = __ldcg(I.meta[1] + w.n1);
    return q;
}
__device__ __forceinline__ RowMeta row_meta(const PatTcArgs& a, const Info& I, const Row& w, const RawMeta& q) {
    RowMeta m;
    const float leaf_u = (a.err ? 8.0f : 2.0f) * kTiny;
    m.E = 0;
    m.fl = w.fl;
    m.er0 = leaf_u;
    m.er1 = I.nch > 1 ? leaf_u : 0.0f;
    m.fm0 = m.fm1 = 0.0f;
    if (I.meta[0]) {
        m.E += q.q0.x >> 2;
        m.fl |= q.q0.x & 3;
        m.er0 = __int_as_float(q.q0.y) + (float)(8 * a.W) * kTiny;
        m.fm0 = fmaxf(__int_as_float(q.q0.z), __int_as_float(q.q0.w));
    }
    if (I.nch > 1 && I.meta[1]) {
        m.E += q.q1.x >> 2;
        m.fl |= q.q1.x & 3;
        m.er1 = __int_as_float(q.q1.y) + (float)(8 * a.W) * kTiny;
        m.fm1 = fmaxf(__int_as_float(q.q1.z), __int_as_float(q.q1.w));
    }
    return m;
}

__device__ __forceinline__ float4 load4(const float* p, int col) { return __ldcg(reinterpret_cast<const float4*>(p + col)); }
__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}

// How a row is scaled, from its statistics: the factors of both children
// before the product (s0, s1), and after it (post).
struct Scale {
    float s0, s1, post;
    int E;
    bool need, nflag;
};

__device__ __forceinline__ int maxexp4(int m, const float4& a, const float4& b) {
    m = max(m, bexp(a.x) + bexp(b.x));
    m = max(m, bexp(a.y) + bexp(b.y));
    m = max(m, bexp(a.z) + bexp(b.z));
    return max(m, bexp(a.w) + bexp(b.w));
}

__device__ __forceinline__ void scale_apart(Scale& s, int maxe, int Eacc) {
    if (maxe < -250) {
        s.nflag = true;
        maxe = 0;
    }
    const int sh = -maxe, part = sh / 2;
    s.s0 = pow2f(part + (sh - part * 2));
    s.s1 = pow2f(part);
    s.E = Eacc + maxe;
}

__device__ __forceinline__ float4 scaled4(const Scale& s, const float4& a, const float4& b) {
    float4 p;
    p.x = (a.x * s.s0) * (b.x * s.s1) * s.post;
    p.y = (a.y * s.s0) * (b.y * s.s1) * s.post;
    p.z = (a.z * s.s0) * (b.z * s.s1) * s.post;
    p.w = (a.w * s.s0) * (b.w * s.s1) * s.post;
    return p;
}

// hi = tf32(v), lo = tf32(v - hi) of four columns into row r's 16-byte piece l
// of an operand chunk (128-byte swizzle).
__device__ __forceinline__ void split_store(float* hi, float* lo, int r, int l, const float4& v) {
    float4 a, b;
    a.x = tc::round_tf32_bits(v.x);
    a.y = tc::round_tf32_bits(v.y);
    a.z = tc::round_tf32_bits(v.z);
    a.w = tc::round_tf32_bits(v.w);
    // (the operand's 13 low bits are ignored: the rounding needs no mask here)
    b.x = __uint_as_float(__float_as_uint(v.x - a.x) + 0x1000u);
    b.y = __uint_as_float(__float_as_uint(v.y - a.y) + 0x1000u);
    b.z = __uint_as_float(__float_as_uint(v.z - a.z) + 0x1000u);
    b.w = __uint_as_float(__float_as_uint(v.w - a.w) + 0x1000u);
    const int at = r * KC + ((l ^ (r & 7)) << 2);
    *reinterpret_cast<float4*>(hi + at) = a;
    *reinterpret_cast<float4*>(lo + at) = b;
}

// The stored row's exponent, flags and error bound (x and y of its record).
__device__ __forceinline__ int2 row_record(const Info& I, const RowMeta& m, const RowStat& t, const Scale& s, bool fused,
                                           bool dead) {
    float u0 = m.er0, u1 = m.er1;
    if (!I.meta[0] && !(t.fmn0 < 0x1p-100f)) u0 = 0.0f;
    if (!I.meta[1] && !(t.fmn1 < 0x1p-100f)) u1 = 0.0f;
    // (a row scaled after the product: its bound scales alike, and a value below
    // 2^-126 before the scaling was flushed)
    const float k0 = s.s0 * s.post;
    u0 *= k0;
    u1 *= s.s1;
    const float ev = u0 * (t.fmx1 * s.s1 + u1) + u1 * (t.fmx0 * k0);
    const float flush = fused && !s.need && s.post != 1.0f ? kTiny * s.post : kTiny;
    int fl = m.fl | (s.nflag ? kFlag : 0);
    if (dead || (fl & kDead)) fl = kDead;
    return make_int2((int)((unsigned)s.E << 2) | fl, __float_as_int(fminf(ev + flush, 1e30f)));
}

// The largest prior-weighted value over root rows 1..Rf and its state (the
// first one), and the largest error bound.
struct Best {
    float f, err;
    int s;
};
struct RootRow {
    float s0, s1, er0, er1;   // the factors' scales and error bounds
    int Rf;
};
template <bool SC>
__device__ __forceinline__ void best_add(Best& b, const RootRow& w, bool leaf0, bool leaf1, float q, int s, float r0,
                                         float r1) {
    if (s > w.Rf) q = 0.0f;
    const float f0 = SC ? r0 * w.s0 : r0, f1 = SC ? r1 * w.s1 : r1;
    const float v = (f0 * f1) * q;
    if (v > b.f) {
        b.f = v;
        b.s = s;
    }
    float u0 = leaf0 && !(r0 < 0x1p-100f) ? 0.0f : w.er0, u1 = leaf1 && !(r1 < 0x1p-100f) ? 0.0f : w.er1;
    if (SC) {
        u0 *= w.s0;
        u1 *= w.s1;
    }
    b.err = fmaxf(b.err, (u0 * (f1 + u1) + u1 * f0) * q);
}
template <bool SC>
__device__ __forceinline__ void best_add4(Best& b, const RootRow& w, bool leaf0, bool leaf1, const float* prior_s, int s,
                                          const float4& x, const float4& y) {
    const float4 q = *reinterpret_cast<const float4*>(prior_s + s);
    best_add<SC>(b, w, leaf0, leaf1, q.x, s, x.x, y.x);
    best_add<SC>(b, w, leaf0, leaf1, q.y, s + 1, x.y, y.y);
    best_add<SC>(b, w, leaf0, leaf1, q.z, s + 2, x.z, y.z);
    best_add<SC>(b, w, leaf0, leaf1, q.w, s + 3, x.w, y.w);
}
__device__ __forceinline__ void best_reduce(Best& b) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float f = __shfl_xor_sync(0xffffffffu, b.f, o), e = __shfl_xor_sync(0xffffffffu, b.err, o);
        const int s = __shfl_xor_sync(0xffffffffu, b.s, o);
        b.err = fmaxf(b.err, e);
        if (f > b.f || (f == b.f && s < b.s)) {      // a tie goes to the first in state order
            b.f = f;
            b.s = s;
        }
    }
}
// Largest product / sum of binary exponents over root rows of a lane's columns.
__device__ __forceinline__ float root_max4(float m, int s, int Rf, const float4& x, const float4& y) {
    if (s >= 1 && s <= Rf) m = fmaxf(m, x.x * y.x);
    if (s + 1 <= Rf) m = fmaxf(m, x.y * y.y);
    if (s + 2 <= Rf) m = fmaxf(m, x.z * y.z);
    if (s + 3 <= Rf) m = fmaxf(m, x.w * y.w);
    return m;
}
__device__ __forceinline__ int root_exp4(int m, int s, int Rf, const float4& x, const float4& y) {
    if (s >= 1 && s <= Rf) m = max(m, bexp(x.x) + bexp(y.x));
    if (s + 1 <= Rf) m = max(m, bexp(x.y) + bexp(y.y));
    if (s + 2 <= Rf) m = max(m, bexp(x.z) + bexp(y.z));
    if (s + 3 <= Rf) m = max(m, bexp(x.w) + bexp(y.w));
    return m;
}

// NCH: 32-column chunks of the bin (1 or 2: every chunk of a unit is
// resident), or 0: any width, two passes over the rows and a ring of two
// stages.
template <int NCH>
struct Shape {
    static constexpr int kDataWarps = NCH == 1 ? 4 : 8;
    static constexpr int kData = 32 * kDataWarps;
    static constexpr int kThreads = kData + 64;
    static constexpr int kStages = NCH ? NCH : 2;
    static constexpr int kPerSm = NCH == 1 ? 4 : NCH == 2 ? 2 : 1;
};

// Floats of one stage: A hi, A lo, B hi, B lo. With resident chunks the B
// area is also the home of the epilogue's 128-row staging tile, so that A is
// free for the next unit's rows as soon as the MMAs are done.
__host__ __device__ inline int stage_floats(int W, int Ns) {
    const int b = 2 * Ns * KC;
    return 2 * kChunkA + (W <= 64 && b < kChunkA ? kChunkA : b);
}

template <int NCH>
struct alignas(16) Shared {
    // (stored is per unit in hand: a warp without rows of a root unit may be done
    // with the next root unit before the others are with this one)
    uint64_t ready[NB], freed[NB], stored[NB], a_full[2], b_full[2], empty[2], mma, a_free, drain;
    uint32_t tmem;
    int abort;
    Info info[NB];
    alignas(16) float prior_s[NCH ? NCH * KC : 512];      // prior of the root size that state s stands for (0 at s = 0)
    long long seg0[kSegSh];
    PatTcNode nodes[kNodeSh];
};

// A wait that gives up when the CTA does. The data warps use the warp-wide
// form below: a warp's lanes go on or give up together.
// Each poll may suspend the thread for up to 10 us (spinning instead would take
// issue slots from the warps that work).
template <class Sh>
__device__ __forceinline__ bool wait_bar(Sh& sh, uint64_t* b, uint32_t parity, int limit = kBarPolls) {
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(tc::smem_u32(b)), "r"(parity), "r"(10000u)
            : "memory");
        if (ok) return true;
        if (*(volatile int*)&sh.abort) return false;
    }
    return false;
}
__device__ __forceinline__ bool test_bar(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(tc::smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
template <class Sh>
__device__ __forceinline__ bool wait_warp(Sh& sh, uint64_t* b, uint32_t parity, int limit = kBarPolls) {
    const bool ok = __all_sync(0xffffffffu, wait_bar(sh, b, parity, limit));
    if (!ok) *(volatile int*)&sh.abort = 1;
    return ok;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(b)) : "memory");
}
// A finished-units count, read once / waited for.
__device__ __forceinline__ int count_now(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool wait_count(const int32_t* p, int n, const int32_t* status, const int* abort) {
    for (int i = 0; i < kPolls; ++i) {
        if (count_now(p) >= n) return true;
        if ((i & 15) == 15 && (*(const volatile int32_t*)status || *(const volatile int*)abort)) return false;
        __nanosleep(64);
    }
    return false;
}

template <class Sh>
__device__ __forceinline__ PatTcNode get_node(const PatTcArgs& a, const Sh& sh, int i) {
    return i < kNodeSh ? sh.nodes[i] : a.nodes[i];
}

// The last of positions lo .. hi - 1 (hi > lo) whose key is at most x, the
// keys ascending from key(lo) <= x: 32 at a time over the warp.
template <class Key>
__device__ __forceinline__ int last_at_most(int lo, int hi, long long x, int lane, Key key) {
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32;
        const int p = lo + lane * step;
        const unsigned m = __ballot_sync(0xffffffffu, p < hi && key(p) <= x);
        lo += (31 - __clz(m)) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// Takes the next unit and fills in its Info (no waits: indices and pointers
// only). Collective over the scheduler warp; false when there is none left.
template <class Sh>
__device__ __forceinline__ bool prepare(const PatTcArgs& a, Sh& sh, Info& I, unsigned long long& next, int lane) {
    const long long idx = (long long)__shfl_sync(0xffffffffu, next, 0);
    if (idx >= a.total_units) return false;
    if (lane == 0) next = atomicAdd(a.next, 1ull);
    const PatTcSeg sg = a.segs[last_at_most(0, a.n_segs, idx, lane, [&](int i) {
        return i < kSegSh ? sh.seg0[i] : a.segs[i].unit0;
    })];
    const int rem = (int)(idx - sg.unit0);
    const int ul = rem / sg.nq;
    const int q = sg.q0 + rem % sg.nq;
    const int k = __ldg(a.active + q), slot = q % a.n_slots;
    const int di = last_at_most(sg.node0, sg.node1, ul, lane, [&](int i) {
        return (long long)(i < kNodeSh ? sh.nodes[i].unit0 : a.nodes[i].unit0);
    });
    const PatTcNode nd = get_node(a, sh, di);
    const int un = ul - nd.unit0;
    const bool is_root = di == a.n_desc - 1;
    const int share = is_root ? 0 : un % a.n_share, p0 = (is_root ? un : un / a.n_share) * TM;
    const int np = min(TM, nd.rows - p0);
    // the rows' child indices
    int i0[TM / 32], i1[TM / 32];
#pragma unroll
    for (int i = 0; i < TM / 32; ++i) {
        const int32_t* ci = a.child + nd.cidx + (int64_t)(p0 + min(lane + 32 * i, np - 1)) * nd.nch;
        i0[i] = __ldg(ci);
        i1[i] = nd.nch > 1 ? __ldg(ci + 1) : 0;
    }
    const int32_t* mi = a.mat_index + (size_t)k * a.n_nodes;
    const int64_t slot_row = (int64_t)slot * a.slot_rows;
    const int m_own = is_root ? 0 : __ldg(mi + nd.node);
    const int m0 = __ldg(mi + nd.child_node[0]), m1 = nd.nch > 1 ? __ldg(mi + nd.child_node[1]) : 0;
    if (lane < 2) {
        const int d = lane < nd.nch ? nd.child[lane] : -1;
        const int m = lane ? m1 : m0;
        if (lane >= nd.nch) {      // no second child: a factor of 1 (and not a leaf)
            I.tab[lane] = g_one_row;
            I.meta[lane] = a.meta;
            I.pitch[lane] = 0;
        } else if (d >= 0) {
            const int64_t r = slot_row + get_node(a, sh, d).row0;
            I.tab[lane] = a.table + r * a.W;
            I.meta[lane] = a.meta + r;
            I.pitch[lane] = a.W;
        } else {
            I.tab[lane] = a.mat_tr + (size_t)(m & ~kSatBit) * a.Wm * a.Wm;
            I.meta[lane] = nullptr;
            I.pitch[lane] = a.Wm;
        }
    }
    if (lane == 0) {
        I.nch = nd.nch;
        I.np = np;
        I.is_root = is_root;
        I.sat = ((m0 | m1) & kSatBit) != 0;
        I.k = k;
        I.stop = 0;
        I.q = q;
        I.di = di;
        I.row_out = (int)(slot_row + nd.row0 + p0);
        I.s_off = share * a.Ns;
        I.mat = m_own & ~kSatBit;
        // (only the unit of a row's first states writes its record)
        I.meta_out = is_root || share ? nullptr : a.meta + slot_row + nd.row0 + p0;
        I.item0 = nd.perm0 + p0;
    }
#pragma unroll
    for (int i = 0; i < TM / 32; ++i) {
        I.idx[0][lane + 32 * i] = i0[i];
        I.idx[1][lane + 32 * i] = i1[i];
    }
    __syncwarp();
    return true;
}

// Waits until everything the unit reads is complete.
template <class Sh>
__device__ __forceinline__ bool wait_inputs(const PatTcArgs& a, const Sh& sh, const Info& I, int lane) {
    bool ok = true;
    const int32_t* p = nullptr;
    int n = 0;
    if (lane < 2 && lane < I.nch) {
        const int d = get_node(a, sh, I.di).child[lane];
        if (d >= 0) {
            p = a.done + (size_t)I.q * a.n_desc + d;
            n = get_node(a, sh, d).n_units;
        }
    } else if (lane == 2 && I.q >= a.n_slots) {      // the table's last user
        p = a.done + (size_t)(I.q - a.n_slots) * a.n_desc + a.n_desc - 1;
        n = get_node(a, sh, a.n_desc - 1).n_units;
    }
    if (p) ok = wait_count(p, n, a.status, &sh.abort);
    ok = __all_sync(0xffffffffu, ok);
    __syncwarp();
    return ok;
}

// The scheduler warp: units into the Info buffers, each handed on once its
// inputs are complete.
template <int NCH>
__device__ void schedule(const PatTcArgs& a, Shared<NCH>& sh, int lane) {
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(a.next, 1ull);
    uint32_t use = 0;            // uses of the buffers so far
    for (int buf = 0;; buf = buf + 1 == NB ? 0 : buf + 1, ++use) {
        bool ok = use < NB || wait_warp(sh, &sh.freed[buf], (use / NB - 1) & 1);
        Info& I = sh.info[buf];
        bool more = false;
        if (ok) {
            more = prepare(a, sh, I, next, lane);
            if (more && !(ok = wait_inputs(a, sh, I, lane)) && lane == 0) {
                atomicCAS(a.status, 0, 1);
                *(volatile int*)&sh.abort = 1;
            }
        }
        if (lane == 0) {
            if (!ok || !more) I.stop = 1;
            mbar_arrive(&sh.ready[buf]);
        }
        if (!ok || !more) return;
    }
}

// The issuer warp (lane 0): matrix chunks by TMA, MMAs, factor tables by TMA,
// and the count of finished units.
template <int NCH>
__device__ void issue(const PatTcArgs& a, const CUtensorMap* map_mat, const CUtensorMap* map_vst,
                      const CUtensorMap* map_vst32, Shared<NCH>& sh, float* stages) {
    constexpr int NST = Shape<NCH>::kStages;
    const int n_chunks = a.W / KC;
    const int sf = stage_floats(a.W, a.Ns);
    const uint32_t idesc = tc::idesc_tf32(TM, a.Ns);
    uint32_t g = 0;              // chunks so far
    int pending_b = 0;           // B loads not yet waited for (bit per stage)
    uint32_t par_b[2] = {0, 0};
    uint32_t use = 0;
    bool ok = true;
    for (int buf = 0; ok; buf = buf + 1 == NB ? 0 : buf + 1, ++use) {
        ok = wait_bar(sh, &sh.ready[buf], (use / NB) & 1);
        if (!ok) break;
        const Info& I = sh.info[buf];
        if (I.stop) break;
        const int np = I.np, q = I.q, di = I.di, row_out = I.row_out, s_off = I.s_off, mat_row = I.mat * a.Wm + s_off;
        const bool is_root = I.is_root;
        if (!is_root) {
            // matrix chunks into the stages: the previous unit's MMAs are done, and
            // its stores have read their staging tiles (waited for below)
            auto load_b = [&](int c) {
                const int st = (int)((g + (uint32_t)c) % NST);
                tc::mbar_expect_tx(&sh.b_full[st], (uint32_t)(2 * a.Ns * KC * sizeof(float)));
                tc::tma_load_3d(stages + (size_t)st * sf + 2 * kChunkA, map_mat, c * KC, mat_row, 0, &sh.b_full[st]);
                pending_b |= 1 << st;
                par_b[st] = ((g + (uint32_t)c) / NST) & 1;
            };
            for (int c = 0; c < NST && c < n_chunks; ++c) load_b(c);
            for (int c = 0; c < n_chunks && ok; ++c) {
                const uint32_t cg = g + (uint32_t)c;
                const int st = (int)(cg % NST);
                const uint32_t par = (cg / NST) & 1;
                ok = wait_bar(sh, &sh.a_full[st], par) && wait_bar(sh, &sh.b_full[st], par);
                if (!ok) break;
                pending_b &= ~(1 << st);
                tc::fence_after();
                const float* Ah = stages + (size_t)st * sf;
                const float* Al = Ah + kChunkA;
                const float* Bh = Al + kChunkA;
                const float* Bl = Bh + a.Ns * KC;
#pragma unroll
                for (int ks = 0; ks < KC / 8; ++ks) {
                    const uint64_t ah = tc::desc_sw128(Ah + ks * 8), al = tc::desc_sw128(Al + ks * 8);
                    const uint64_t bh = tc::desc_sw128(Bh + ks * 8), bl = tc::desc_sw128(Bl + ks * 8);
                    tc::mma_tf32(sh.tmem, ah, bh, idesc, (c == 0 && ks == 0) ? 0u : 1u);
                    tc::mma_tf32(sh.tmem, ah, bl, idesc, 1);
                    tc::mma_tf32(sh.tmem, al, bh, idesc, 1);
                }
                if (NCH == 0) tc::mma_commit(&sh.empty[st]);
                if (c + 1 == n_chunks) tc::mma_commit(&sh.mma);
                // the stage of the chunk before is free when its MMAs are done
                if (NCH == 0 && c >= 1 && c - 1 + NST < n_chunks) {
                    const uint32_t pg = cg - 1;
                    ok = wait_bar(sh, &sh.empty[pg % NST], (pg / NST) & 1);
                    if (ok) load_b(c - 1 + NST);
                }
            }
            g += (uint32_t)n_chunks;
        }
        ok = ok && wait_bar(sh, &sh.stored[buf], (use / NB) & 1);
        if (!ok) break;
        mbar_arrive(&sh.freed[buf]);       // nobody reads this unit's Info any more
        if (!is_root) {
            for (int c = 0; c < a.Ns / KC; ++c) {
                float* t = NCH ? stages + (size_t)c * sf + 2 * kChunkA : stages + (size_t)c * kChunkA;
                if (np > TM - 32) {
                    tc::tma_store_2d(map_vst, s_off + c * KC, row_out, t);
                } else {
                    for (int r = 0; r < np; r += 32) tc::tma_store_2d(map_vst32, s_off + c * KC, row_out + r, t + r * KC);
                }
            }
            tc::bulk_commit();
            tc::bulk_wait_read0();
            if (NCH == 0) mbar_arrive(&sh.a_free);
            tc::bulk_wait0();
            tc::fence_proxy_async_global();
        }
        __threadfence();
        atomicAdd(a.done + (size_t)q * a.n_desc + di, 1);
    }
    if (!ok) {
        // some wait of this CTA gave up
        atomicCAS(a.status, 0, 1);
        *(volatile int*)&sh.abort = 1;
    }
    // drain: loads of ours still landing, MMAs still running
    for (int q = 0; q < NST; ++q)
        if (pending_b >> q & 1) tc::mbar_wait(&sh.b_full[q], par_b[q], 1 << 20);
    tc::mma_commit(&sh.drain);
    tc::mbar_wait(&sh.drain, 0, 1 << 24);
    tc::bulk_wait0();
}

// Rows of a unit go to the data warps in groups of four, eight lanes a row:
// group i of warp w holds rows 4 (i DW + w) .. + 3, so a short tile's rows
// spread over the warps and its missing ones cost nothing. What is done once
// per row (pointers, records, the root's logarithm) is done by the row's owner
// lane 4 i + (row & 3), for all of a warp's rows at once.
template <int NCH>
__device__ void data(const PatTcArgs& a, Shared<NCH>& sh, float* stages, int tid) {
    constexpr int DW = Shape<NCH>::kDataWarps, NST = Shape<NCH>::kStages;
    constexpr int GPW = TM / 4 / DW;      // groups per warp
    constexpr int VC = NCH ? NCH : 1;
    const int warp = tid >> 5, lane = tid & 31, l = lane & 7, sub = lane >> 3;
    const int n_chunks = NCH ? NCH : a.W / KC;
    const int sf = stage_floats(a.W, a.Ns);
    const bool fused = a.W <= 64;         // rows of up to 64 states are scaled after the product
    const int own = lane < 4 * GPW ? 4 * ((lane >> 2) * DW + warp) + (lane & 3) : TM;   // the row this lane owns
    const int from = (lane & 3) * 8;      // a lane of the eight that work on it (in its group's turn)
    uint32_t g = 0, gu = 0;               // chunks and GEMM units so far
    // the unit being worked on; the next one's is set up (and its first loads
    // issued) while this one's GEMM runs
    const Info* Ip = nullptr;
    bool leaf0 = false, leaf1 = false;
    int np = 0, groups = 0;
    Row w{0, 0, 0};
    RawMeta raw;
    const float *t0 = nullptr, *t1 = nullptr;      // this lane's columns of the children's row 0
    unsigned pitch0 = 0, pitch1 = 0;
    auto row0 = [&](int src) { return t0 + (size_t)pitch0 * (unsigned)__shfl_sync(0xffffffffu, w.n0, src); };
    auto row1 = [&](int src) { return t1 + (size_t)pitch1 * (unsigned)__shfl_sync(0xffffffffu, w.n1, src); };
    // Resident chunks: all of a unit's factors are copied into the operand
    // area, a lane's 16-byte pieces of the first child where their product's hi
    // part will be, of the second where its lo part will be. A lane reads back
    // only what it copied.
    auto piece = [&](int i, int c) {
        const int r = 4 * (i * DW + warp) + sub;
        return stages + (size_t)c * sf + r * KC + ((l ^ (r & 7)) << 2);
    };
    auto copy_rows = [&]() {
        for (int i = 0; i < groups; ++i) {
            const float* p0 = row0(4 * i + sub);
            const float* p1 = row1(4 * i + sub);
#pragma unroll
            for (int c = 0; c < VC; ++c) {
                cp16(piece(i, c), p0 + c * KC);
                cp16(piece(i, c) + kChunkA, p1 + c * KC);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float4 x[VC], y[VC];      // the group's factors
    auto get_rows = [&](int i) {
#pragma unroll
        for (int c = 0; c < VC; ++c) {
            x[c] = *reinterpret_cast<const float4*>(piece(i, c));
            y[c] = *reinterpret_cast<const float4*>(piece(i, c) + kChunkA);
        }
    };
    auto begin = [&](const Info& I) {
        Ip = &I;
        leaf0 = !I.meta[0];
        leaf1 = !I.meta[1];
        np = I.np;
        groups = max(0, min(GPW, ((np + 3) / 4 - warp + DW - 1) / DW));   // this warp's (warp-uniform)
        w = make_row(a, I, own);
        t0 = I.tab[0] + 4 * l;
        t1 = I.tab[1] + 4 * l;
        pitch0 = (unsigned)I.pitch[0];
        pitch1 = (unsigned)I.pitch[1];
        if (NCH) copy_rows();
        raw = load_meta(I, own, w);
    };
    bool begun = false;
    uint32_t use = 0;
    for (int buf = 0;; buf = buf + 1 == NB ? 0 : buf + 1, ++use) {
        if (!begun) {
            if (!wait_warp(sh, &sh.ready[buf], (use / NB) & 1)) return;
            if (sh.info[buf].stop) return;
            begin(sh.info[buf]);
        }
        begun = false;
        const Info& I = *Ip;
        if (NCH) asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (I.is_root) {
            const RowMeta m = row_meta(a, I, w, raw);
            const int64_t fam = own < np ? __ldg(a.perm + I.item0 + own) : 0;
            const int Rf_own = own < np ? __ldg(a.item_R + I.item0 + own) : 0;
            const bool check_dead = I.sat && !a.err;
            Best mine{0.0f, 0.0f, 1 << 30};
            float my_s0 = 1.0f, my_s1 = 1.0f, my_max = 1.0f;
            int my_E = m.E;
            bool my_nflag = false;
#pragma unroll 1
            for (int i = 0; i < groups; ++i) {
                const int src = 4 * i + sub;
                if (NCH) get_rows(i);
                RootRow rr;
                rr.s0 = rr.s1 = 1.0f;
                rr.er0 = __shfl_sync(0xffffffffu, m.er0, src);
                rr.er1 = __shfl_sync(0xffffffffu, m.er1, src);
                rr.Rf = __shfl_sync(0xffffffffu, Rf_own, src);
                const float* p0 = row0(src);
                const float* p1 = row1(src);
                Best best{0.0f, 0.0f, 1 << 30};
#pragma unroll(NCH ? NCH : 1)
                for (int c = 0; c < n_chunks; ++c)
                    best_add4<false>(best, rr, leaf0, leaf1, sh.prior_s, c * KC + 4 * l,
                                     NCH ? x[NCH ? c : 0] : load4(p0, c * KC), NCH ? y[NCH ? c : 0] : load4(p1, c * KC));
                best_reduce(best);
                const bool mine_now = (lane >> 2) == i;
                if (check_dead) {
                    float mp = 0.0f;
                    for (int c = 0; c < n_chunks; ++c)
                        mp = root_max4(mp, c * KC + 4 * l, rr.Rf, load4(p0, c * KC), load4(p1, c * KC));
                    mp = __shfl_sync(0xffffffffu, lane8_max(mp), from);
                    if (mine_now) my_max = mp;
                }
                const bool need = 4 * (i * DW + warp) + sub < np && !(best.f > 0.0f);
                if (__any_sync(0xffffffffu, need)) {
                    // the product underflows at every root row: the factors scaled apart
                    int maxe = -100000;
                    for (int c = 0; c < n_chunks; ++c)
                        maxe = root_exp4(maxe, c * KC + 4 * l, rr.Rf, load4(p0, c * KC), load4(p1, c * KC));
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) maxe = max(maxe, __shfl_xor_sync(0xffffffffu, maxe, o));
                    Scale sc{1.0f, 1.0f, 1.0f, 0, need, false};
                    if (need) scale_apart(sc, maxe, 0);
                    rr.s0 = sc.s0;
                    rr.s1 = sc.s1;
                    best = Best{0.0f, 0.0f, 1 << 30};
                    for (int c = 0; c < n_chunks; ++c)
                        best_add4<true>(best, rr, leaf0, leaf1, sh.prior_s, c * KC + 4 * l, load4(p0, c * KC), load4(p1, c * KC));
                    best_reduce(best);
                    const float t0 = __shfl_sync(0xffffffffu, sc.s0, from), t1 = __shfl_sync(0xffffffffu, sc.s1, from);
                    const int tE = __shfl_sync(0xffffffffu, sc.E, from), tn = __shfl_sync(0xffffffffu, (int)sc.nflag, from);
                    if (mine_now) {
                        my_s0 = t0;
                        my_s1 = t1;
                        my_E += tE;
                        my_nflag = tn != 0;
                    }
                }
                const float f = __shfl_sync(0xffffffffu, best.f, from), e = __shfl_sync(0xffffffffu, best.err, from);
                const int s = __shfl_sync(0xffffffffu, best.s, from);
                if (mine_now) mine = Best{f, e, s};
            }
            if (own < np) {
                const bool dead = (m.fl & kDead) || (check_dead && !(my_max > 0.0f));
                bool flag = ((m.fl & kFlag) || my_nflag) && !dead;
                double o = NAN;
                float p = 0.0f, q = 0.0f;
                if (mine.f > 0.0f) {
                    p = (__ldcg(I.tab[0] + (size_t)pitch0 * (unsigned)w.n0 + mine.s) * my_s0) *
                        (__ldcg(I.tab[1] + (size_t)pitch1 * (unsigned)w.n1 + mine.s) * my_s1);
                    q = sh.prior_s[mine.s];
                }
                const double best = (double)p * (double)q;
                if (dead) o = a.model == 0 ? -INFINITY : NAN;   // log 0 (base) / a failed family (gamma)
                else if (best > 0.0 && !flag)
                    o = log(best * a.cat_probs[I.k]) + (double)my_E * 0.69314718055994530942;
                else flag = true;
                a.out[(size_t)fam * a.K + I.k] = o;
                a.out_err[(size_t)fam * a.K + I.k] = (dead || flag || !(mine.f > 0.0f)) ? 0.0f : mine.err / mine.f;
                if (flag) {
                    atomicOr(&a.flags[fam], 1);
                    a.term_flags[(size_t)fam * a.K + I.k] = 1;   // this category term
                    atomicOr(a.any_flag, 1);
                }
            }
            __syncwarp();
            mbar_arrive(&sh.stored[buf]);
            continue;
        }

        // ---- rows: product, scaling, TF32 operands ----
        RowStat st;                    // of the row this lane owns
        stat_init(st);
        st.maxp = 1.0f;
        Scale ms{1.0f, 1.0f, 1.0f, 0, false, false};
        // the scales of group i's rows, from their statistics (warp-collective;
        // X, Y give a lane's columns of chunk c)
        auto scales = [&](int i, RowStat t, auto X, auto Y) {
            const int r = 4 * (i * DW + warp) + sub;
            const bool mine_now = (lane >> 2) == i;
            Scale sc{1.0f, 1.0f, 1.0f, 0, r < np && !(t.maxp >= 0x1p-120f), false};
            // (rows that keep their scale take none of this)
            if (__any_sync(0xffffffffu, r < np && !(t.maxp >= 0x1p-32f))) {
                if (!sc.need && t.maxp > 0.0f && t.maxp < 0x1p-32f) {
                    // bring this row's maximum back to [0.5, 1): after the product for
                    // rows of up to 64 states, before it for wider ones
                    const int kk = -bexp(t.maxp);
                    (fused ? sc.post : sc.s0) = pow2f(kk);
                    sc.E = -kk;
                }
                if (__any_sync(0xffffffffu, sc.need)) {
                    int maxe = -100000;
                    #pragma unroll(NCH ? NCH : 1)
                    for (int c = 0; c < n_chunks; ++c) maxe = maxexp4(maxe, X(c), Y(c));
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) maxe = max(maxe, __shfl_xor_sync(0xffffffffu, maxe, o));
                    if (sc.need) scale_apart(sc, maxe, 0);
                }
                const float t0 = __shfl_sync(0xffffffffu, sc.s0, from), t1 = __shfl_sync(0xffffffffu, sc.s1, from);
                const float tp = __shfl_sync(0xffffffffu, sc.post, from);
                const int tE = __shfl_sync(0xffffffffu, sc.E, from);
                const int tn = __shfl_sync(0xffffffffu, (sc.need ? 1 : 0) | (sc.nflag ? 2 : 0), from);
                if (mine_now) ms = Scale{t0, t1, tp, tE, (tn & 1) != 0, (tn & 2) != 0};
            }
            const float mp = __shfl_sync(0xffffffffu, t.maxp, from);
            if (mine_now) st.maxp = mp;
            return sc;
        };
        // a leaf's largest and smallest factor go to the row's owner
        auto leaf_stat = [&](int i, bool second, float mx, float mn) {
            mx = __shfl_sync(0xffffffffu, lane8_max(mx), from);
            mn = __shfl_sync(0xffffffffu, lane8_min(mn), from);
            if ((lane >> 2) == i) {
                (second ? st.fmx1 : st.fmx0) = mx;
                (second ? st.fmn1 : st.fmn0) = mn;
            }
        };
        if (NCH) {
#pragma unroll 2
            for (int i = 0; i < groups; ++i) {
                get_rows(i);
                const int r = 4 * (i * DW + warp) + sub;
                float4 pr[VC];
                RowStat t;
                t.maxp = 0.0f;
#pragma unroll
                for (int c = 0; c < VC; ++c) {
                    pr[c] = make_float4(x[c].x * y[c].x, x[c].y * y[c].y, x[c].z * y[c].z,
                                        x[c].w * y[c].w);
                    t.maxp = fmaxf(t.maxp, max4(pr[c]));
                }
                if (leaf0) {
                    float mx = max4(x[0]), mn = min4(x[0]);
#pragma unroll
                    for (int c = 1; c < VC; ++c) {
                        mx = fmaxf(mx, max4(x[c]));
                        mn = fminf(mn, min4(x[c]));
                    }
                    leaf_stat(i, false, mx, mn);
                }
                if (leaf1) {
                    float mx = max4(y[0]), mn = min4(y[0]);
#pragma unroll
                    for (int c = 1; c < VC; ++c) {
                        mx = fmaxf(mx, max4(y[c]));
                        mn = fminf(mn, min4(y[c]));
                    }
                    leaf_stat(i, true, mx, mn);
                }
                // rows whose maximum is at least 2^-32 keep their scale: one of a row's
                // eight lanes saw it
                unsigned big = __ballot_sync(0xffffffffu, t.maxp >= 0x1p-32f || r >= np);
                big |= big >> 1;
                big |= big >> 2;
                big |= big >> 4;
                if ((big & 0x01010101u) != 0x01010101u) {
                    t.maxp = lane8_max(t.maxp);
                    const Scale sc = scales(i, t, [&](int c) { return x[c]; }, [&](int c) { return y[c]; });
#pragma unroll
                    for (int c = 0; c < VC; ++c) pr[c] = scaled4(sc, x[c], y[c]);
                }
#pragma unroll
                for (int c = 0; c < VC; ++c)
                    split_store(stages + (size_t)c * sf, stages + (size_t)c * sf + kChunkA, r, l, pr[c]);
            }
            tc::fence_proxy_async_shared();
            for (int c = 0; c < NCH; ++c) mbar_arrive(&sh.a_full[c]);
        } else {
            // statistics first, then the operands chunk by chunk (the rows' second
            // read comes from L2)
            const float *q0[GPW], *q1[GPW];
            Scale sc[GPW];
#pragma unroll
            for (int i = 0; i < GPW; ++i) {
                q0[i] = row0(4 * i + sub);
                q1[i] = row1(4 * i + sub);
                if (i >= groups) continue;
                RowStat t;
                stat_init(t);
#pragma unroll 4
                for (int c = 0; c < n_chunks; ++c) stat_add4(t, load4(q0[i], c * KC), load4(q1[i], c * KC));
                t.maxp = lane8_max(t.maxp);
                leaf_stat(i, false, t.fmx0, t.fmn0);
                leaf_stat(i, true, t.fmx1, t.fmn1);
                sc[i] = scales(i, t, [&](int c) { return load4(q0[i], c * KC); }, [&](int c) { return load4(q1[i], c * KC); });
            }
            if (gu && !wait_warp(sh, &sh.a_free, (gu - 1) & 1)) return;
            for (int c = 0; c < n_chunks; ++c) {
                const uint32_t cg = g + (uint32_t)c;
                const int stg = (int)(cg % NST);
                float4 u[GPW], v[GPW];
#pragma unroll
                for (int i = 0; i < GPW; ++i) {
                    if (i >= groups) continue;
                    u[i] = load4(q0[i], c * KC);
                    v[i] = load4(q1[i], c * KC);
                }
                if (c >= NST && !wait_warp(sh, &sh.empty[stg], (cg / NST - 1) & 1)) return;
                float* Ah = stages + (size_t)stg * sf;
#pragma unroll
                for (int i = 0; i < GPW; ++i) {
                    if (i >= groups) continue;
                    split_store(Ah, Ah + kChunkA, 4 * (i * DW + warp) + sub, l, scaled4(sc[i], u[i], v[i]));
                }
                tc::fence_proxy_async_shared();
                mbar_arrive(&sh.a_full[stg]);
            }
            g += (uint32_t)n_chunks;
        }
        // the owned row's record
        if (I.meta_out && own < np) {
            const RowMeta m = row_meta(a, I, w, raw);
            ms.E += m.E;
            if (NCH && !leaf0) st.fmx0 = m.fm0;
            if (NCH && !leaf1) st.fmx1 = I.nch > 1 ? m.fm1 : 1.0f;
            const bool dead = I.sat && !a.err && !(st.maxp > 0.0f);
            *reinterpret_cast<int2*>(I.meta_out + own) = row_record(I, m, st, ms, fused, dead);
        }

        int4* const out = I.meta_out;
        const int np_out = np;

        // ---- epilogue: factors from TMEM into the staging tiles ----
        // (a test hook can make this wait give up after limit - 1 polls)
        if (!wait_warp(sh, &sh.mma, gu & 1, a.debug_wait_limit > 0 ? a.debug_wait_limit - 1 : kBarPolls)) {
            if (lane == 0) atomicCAS(a.status, 0, 2);
            return;
        }
        tc::fence_after();
        // the operand area is free: the next unit's rows, if its inputs are complete
        const int nb = buf + 1 == NB ? 0 : buf + 1;
        if (NCH && __all_sync(0xffffffffu, test_bar(&sh.ready[nb], ((use + 1) / NB) & 1)) && !sh.info[nb].stop) {
            begin(sh.info[nb]);
            begun = true;
        }
        if (32 * (warp & 3) < np_out) {
            const int row = 32 * (warp & 3) + lane;
            const uint32_t base = sh.tmem + ((uint32_t)(32 * (warp & 3)) << 16);
            for (int c = warp >> 2; c < a.Ns / KC; c += DW / 4) {
                float mx = 0.0f;
                float* t = (NCH ? stages + (size_t)c * sf + 2 * kChunkA : stages + (size_t)c * kChunkA) + row * KC;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[16];
                    tc::tmem_ld16(base + (uint32_t)(c * KC + 16 * h), v);
#pragma unroll
                    for (int q = 0; q < 16; ++q) mx = fmaxf(mx, __uint_as_float(v[q]));
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<uint4*>(t + (((4 * h + q) ^ (row & 7)) << 2)) =
                            make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                if (NCH && row < np_out) {
                    // the factor row's largest value over these columns, for its readers'
                    // error bounds
                    int* o = reinterpret_cast<int*>(out + row) + 2;
                    o[c] = __float_as_int(mx);
                    if (NCH == 1) o[1] = 0;
                }
            }
        }
        tc::fence_before();
        tc::fence_proxy_async_shared();
        mbar_arrive(&sh.stored[buf]);
        ++gu;
    }
}

template <int NCH>
__global__ void __launch_bounds__(Shape<NCH>::kThreads, Shape<NCH>::kPerSm)
    k_pat_tc(const __grid_constant__ CUtensorMap map_mat, const __grid_constant__ CUtensorMap map_vst,
             const __grid_constant__ CUtensorMap map_vst32, const PatTcArgs a) {
    extern __shared__ uint8_t raw[];
    float* stages = reinterpret_cast<float*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    __shared__ Shared<NCH> sh;
    constexpr int ND = Shape<NCH>::kData;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int j = tid; j < (NCH ? NCH * KC : 512); j += ND + 64)
        sh.prior_s[j] = j > 0 && j <= a.n_prior ? (float)a.prior[j - 1] : 0.0f;
    for (int j = tid; j < min(a.n_segs, kSegSh); j += ND + 64) sh.seg0[j] = a.segs[j].unit0;
    for (int j = tid; j < min(a.n_desc, kNodeSh); j += ND + 64) sh.nodes[j] = a.nodes[j];
    if (warp == ND / 32 + 1) tc::tmem_alloc(&sh.tmem, (uint32_t)a.tmem_cols);
    if (tid == 0) {
        for (int q = 0; q < NB; ++q) {
            tc::mbar_init(&sh.ready[q], 1);
            tc::mbar_init(&sh.freed[q], 1);
            tc::mbar_init(&sh.stored[q], ND);
        }
        for (int q = 0; q < 2; ++q) {
            tc::mbar_init(&sh.a_full[q], ND);
            tc::mbar_init(&sh.b_full[q], 1);
            tc::mbar_init(&sh.empty[q], 1);
        }
        tc::mbar_init(&sh.mma, 1);
        tc::mbar_init(&sh.a_free, 1);
        tc::mbar_init(&sh.drain, 1);
        tc::mbar_init_fence();
        sh.abort = 0;
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == ND / 32) {
        schedule<NCH>(a, sh, lane);
    } else if (warp == ND / 32 + 1) {
        if (lane == 0) issue<NCH>(a, &map_mat, &map_vst, &map_vst32, sh, stages);
        __syncwarp();
    } else {
        data<NCH>(a, sh, stages, tid);
    }
    __syncthreads();
    if (warp == ND / 32 + 1) tc::tmem_dealloc(sh.tmem, (uint32_t)a.tmem_cols);
}

template <int NCH>
cudaError_t init_one() {
    return cudaFuncSetAttribute(k_pat_tc<NCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(200 * 1024));
}

size_t dyn_smem(int W, int Ns) {
    const int stages = W == 32 ? 1 : 2;
    // (wide bins: the stages are also home of the epilogue's staging tiles)
    return sizeof(float) * std::max<size_t>((size_t)stages * stage_floats(W, Ns), (size_t)(Ns / KC) * kChunkA) + 1024;
}

}  // namespace

// States of a unit: the whole bin up to 128 states, else equal shares of 96
// or 128 (192 = 2 x 96).
int pat_tc_states(int W) { return W <= 128 ? W : W == 192 ? 96 : 128; }

cudaError_t pat_tc_init() {
    float ones[512];
    for (float& x : ones) x = 1.0f;
    cudaError_t e = cudaMemcpyToSymbol(g_one_row, ones, sizeof ones);
    if (e == cudaSuccess) e = init_one<0>();
    if (e == cudaSuccess) e = init_one<1>();
    return e == cudaSuccess ? init_one<2>() : e;
}

// (The occupancy query counts one CTA per SM for a kernel that allocates
// TMEM, whatever it allocates; what fits is shared memory, registers and the
// 512 TMEM columns.)
int pat_tc_ctas_per_sm(int W) {
    static std::atomic<int> known[17];       // by W / 32 (the same on every device this runs on)
    const int at = std::min(16, W / 32);
    if (const int k = known[at].load()) return k;
    const int Ns = pat_tc_states(W);
    const void* fn = W == 32 ? (const void*)k_pat_tc<1> : W == 64 ? (const void*)k_pat_tc<2> : (const void*)k_pat_tc<0>;
    const int threads = W == 32 ? Shape<1>::kThreads : W == 64 ? Shape<2>::kThreads : Shape<0>::kThreads;
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    int cols = 32;
    while (cols < Ns) cols *= 2;
    const int by_smem = (int)((size_t)228 * 1024 / (dyn_smem(W, Ns) + fa.sharedSizeBytes + 1024));
    const int by_regs = 65536 / ((fa.numRegs + 7) / 8 * 8 * threads);
    const int n = std::max(1, std::min({by_smem, by_regs, 512 / cols}));
    known[at].store(n);
    return n;
}

cudaError_t launch_pat_tc(const PatTcMaps& m, const PatTcArgs& a, int n_ctas, cudaStream_t s) {
    if (a.total_units <= 0) return cudaSuccess;
    if (a.W % 32 || a.W > 512 || a.Ns != pat_tc_states(a.W) || a.Ns * a.n_share != a.W || a.tmem_cols < a.Ns)
        return cudaErrorInvalidValue;
    const size_t sm = dyn_smem(a.W, a.Ns);
    if (a.W == 32) k_pat_tc<1><<<n_ctas, Shape<1>::kThreads, sm, s>>>(m.mat, m.vst, m.vst32, a);
    else if (a.W == 64) k_pat_tc<2><<<n_ctas, Shape<2>::kThreads, sm, s>>>(m.mat, m.vst, m.vst32, a);
    else k_pat_tc<0><<<n_ctas, Shape<0>::kThreads, sm, s>>>(m.mat, m.vst, m.vst32, a);
    return cudaGetLastError();
}

}  // namespace cafe
