// Distinct count patterns below every internal node of the tree.
//
// A node's vector depends only on the counts of the leaves below it (and on
// the state bound), so families of one group (an S-bin, or the whole set)
// that agree there share it. The reference does this for whole families
// (build_reference_list, src/base_model.cpp:27-51); here every subtree is
// deduplicated, so the pruning kernels contract each distinct row once and
// a parent's row picks its children's rows by index. On gene families most
// subtrees of a few leaves hold a few hundred patterns: 10,000 families of
// 24 taxa have 4.4 times fewer rows than families x nodes, 50,000 of 32
// taxa 4.7 times.
//
// Items are the families in group order. Bottom up, level by level:
//   k_pat_insert   an item's key at a node is its children's keys: a leaf's
//                  count, an internal child's representative item. Open
//                  addressing over item indices; the first item to claim a
//                  slot represents its key (keys are compared through the
//                  representative's own children, so nothing else is stored
//                  and nothing is published late).
//   k_pat_number   representatives of a node get consecutive row numbers in
//                  item order, from 0 in every group.
//   k_pat_counts   marks the counts that occur at every leaf in every group.
//   k_pat_write    every row's child indices: a leaf's count, or the row of
//                  the internal child. The root keeps one row per family.
// Which item represents a key depends on timing; the rows' contents do not.
#include "common.cuh"

#include <algorithm>

namespace cafe {
namespace {

constexpr int kNumberThreads = 1024;

__device__ __forceinline__ int group_of(const PatBuildArgs& a, int64_t i) {
    int lo = 0, hi = a.n_groups;      // the last group whose first item is not past i (empty groups precede it)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(a.group_first + mid) <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The item's key at child `ch`.
__device__ __forceinline__ int32_t child_key(const PatBuildArgs& a, int ch, int64_t item) {
    const int lc = a.plan.leaf_col[ch];
    if (lc >= 0) return a.counts[(size_t)a.perm[item] * a.plan.n_leaves + lc];
    return a.rep[(size_t)a.node_ii[ch] * a.F + item];
}

__global__ void __launch_bounds__(256) k_pat_insert(PatBuildArgs a, const int32_t* __restrict__ nodes, int32_t* table,
                                                    int64_t mask) {
    const int ii = nodes[blockIdx.y];
    int32_t* tab = table + (size_t)blockIdx.y * (mask + 1);
    const int c0 = a.plan.cstart[ii], c1 = a.plan.cstart[ii + 1];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.F; i += (int64_t)gridDim.x * blockDim.x) {
        const int g = group_of(a, i);
        uint64_t h = (uint64_t)(g + 1) * 0x9E3779B97F4A7C15ull;
        for (int c = c0; c < c1; ++c) {
            h ^= (uint64_t)(uint32_t)child_key(a, a.plan.child[c], i);
            h *= 0xC2B2AE3D27D4EB4Full;
            h ^= h >> 29;
        }
        int64_t s = (int64_t)(h >> 7) & mask;
        int32_t owner;
        // the table has at least twice as many slots as items, so the probe ends
        for (;;) {
            // (a slot is written once: reading it first spares the atomics of the many items of a common key)
            owner = *(volatile int32_t*)&tab[s];
            if (owner < 0) owner = atomicCAS(&tab[s], -1, (int32_t)i);
            if (owner < 0) {
                owner = (int32_t)i;
                break;
            }
            bool same = group_of(a, owner) == g;
            for (int c = c0; c < c1 && same; ++c) {
                const int ch = a.plan.child[c];
                same = child_key(a, ch, owner) == child_key(a, ch, i);
            }
            if (same) break;
            s = (s + 1) & mask;
        }
        a.rep[(size_t)ii * a.F + i] = owner;
    }
}

// One block per node: exclusive count of representatives
// before each item, and its value at every group's first item.
__global__ void __launch_bounds__(kNumberThreads) k_pat_number(PatBuildArgs a, const int32_t* __restrict__ nodes) {
    __shared__ int wsum[kNumberThreads / 32];
    const int ii = nodes[blockIdx.x];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int32_t* rep = a.rep + (size_t)ii * a.F;
    int32_t* num = a.num + (size_t)ii * a.F;
    int32_t* base = a.base + (size_t)ii * (a.n_groups + 1);
    int total = 0;
    for (int64_t i0 = 0; i0 < a.F; i0 += kNumberThreads) {
        const int64_t i = i0 + tid;
        const bool is = i < a.F && rep[i] == (int32_t)i;
        const unsigned m = __ballot_sync(0xffffffffu, is);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < kNumberThreads / 32; ++w) {
            const int v = wsum[w];
            before += w < warp ? v : 0;
            all += v;
        }
        const int excl = total + before + __popc(m & ((1u << lane) - 1u));
        if (i < a.F) num[i] = excl;
        total += all;
        __syncthreads();
    }
    for (int g = tid; g <= a.n_groups; g += kNumberThreads) {
        const int64_t i = a.group_first[g];
        base[g] = i < a.F ? num[i] : total;
    }
}

__global__ void __launch_bounds__(256) k_pat_write(PatBuildArgs a, const int32_t* __restrict__ nodes,
                                                   const int64_t* __restrict__ child_off, int32_t* out) {
    const int ii = nodes[blockIdx.y];
    const bool is_root = a.plan.internal[ii] == a.plan.root;
    const int c0 = a.plan.cstart[ii], nch = a.plan.cstart[ii + 1] - c0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.F; i += (int64_t)gridDim.x * blockDim.x) {
        if (!is_root && a.rep[(size_t)ii * a.F + i] != (int32_t)i) continue;
        const int g = group_of(a, i);
        const int64_t row = is_root ? i - a.group_first[g]
                                    : a.num[(size_t)ii * a.F + i] - a.base[(size_t)ii * (a.n_groups + 1) + g];
        int32_t* o = out + child_off[(size_t)g * a.plan.n_internal + ii] + row * nch;
        for (int c = 0; c < nch; ++c) {
            const int ch = a.plan.child[c0 + c];
            const int32_t key = child_key(a, ch, i);
            if (a.plan.leaf_col[ch] >= 0) {
                o[c] = key;
            } else {
                const int ci = a.node_ii[ch];
                o[c] = a.num[(size_t)ci * a.F + key] - a.base[(size_t)ci * (a.n_groups + 1) + g];
            }
        }
    }
}

// flags[flag_off[g] + leaf * (group_max[g] + 1) + n]: some family of group g
// has n at the leaf.
__global__ void __launch_bounds__(256) k_pat_counts(PatBuildArgs a, uint8_t* flags) {
    const int nl = a.plan.n_leaves;
    const int64_t total = a.F * nl;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / nl;
        const int c = (int)(e % nl), g = group_of(a, i);
        const int n = a.counts[(size_t)a.perm[i] * nl + c];
        uint8_t* f = flags + a.flag_off[g] + (size_t)c * (a.group_max[g] + 1) + n;
        if (!*(volatile uint8_t*)f) *f = 1;
    }
}

}  // namespace

cudaError_t launch_pat_counts(const PatBuildArgs& a, uint8_t* flags, cudaStream_t s) {
    const int64_t total = a.F * a.plan.n_leaves;
    if (total <= 0) return cudaSuccess;
    k_pat_counts<<<(unsigned)std::min<int64_t>((total + 255) / 256, 4096), 256, 0, s>>>(a, flags);
    return cudaGetLastError();
}

cudaError_t launch_pat_insert(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, int32_t* table, int64_t slots,
                              cudaStream_t s) {
    if (a.F <= 0 || n_nodes <= 0) return cudaSuccess;
    const int bx = (int)std::min<int64_t>((a.F + 255) / 256, 4096);
    k_pat_insert<<<dim3(bx, n_nodes), 256, 0, s>>>(a, d_nodes, table, slots - 1);
    return cudaGetLastError();
}

cudaError_t launch_pat_number(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, cudaStream_t s) {
    if (a.F <= 0 || n_nodes <= 0) return cudaSuccess;
    k_pat_number<<<n_nodes, kNumberThreads, 0, s>>>(a, d_nodes);
    return cudaGetLastError();
}

cudaError_t launch_pat_write(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, const int64_t* d_child_off,
                             int32_t* d_child, cudaStream_t s) {
    if (a.F <= 0 || n_nodes <= 0) return cudaSuccess;
    const int bx = (int)std::min<int64_t>((a.F + 255) / 256, 4096);
    k_pat_write<<<dim3(bx, n_nodes), 256, 0, s>>>(a, d_nodes, d_child_off, d_child);
    return cudaGetLastError();
}

}  // namespace cafe
