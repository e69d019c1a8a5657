// Shared definitions of the GB300 CAFE5 likelihood kernels.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cafe {

// Transition-matrix build job: one (lambda, t) matrix of side `size`,
// computed at the quantized values (matrix_cache_key, src/matrix_cache.h:49-62).
struct MatrixJob {
    double lambda;    // quantized lambda
    double t;         // quantized branch length
    double* dst;      // FP64 row-major size x size, M[parent s][child c]
    float* colT;      // optional: FP32 transposed, column-normalised (size x size), or null
    int32_t* colE;    // optional: per-column power-of-two exponent (size), or null
    uint16_t* hi;     // optional: BF16 hi part, row-major (size x ld_bf16), or null
    uint16_t* lo;     // optional: BF16 lo part
    int size;
    int ld_bf16;      // leading dimension of hi/lo in elements (multiple of 8)
};

// Work tile of the pruning kernels: `count` families (indices into the
// request's family permutation starting at `first`) scored in category `k`
// with state bound S (vectors of S + 1 states) and R root rows starting at
// root size `root_lo` (0 means 1: root sizes 1..R).
struct PruneTile {
    int first;
    int count;
    int k;
    int S;
    int R;
    int root_lo;
    int pad[2];
};

// Flattened tree for the kernels, in one device allocation.
//   internal[i]                internal nodes in post-order (root last)
//   cstart[i]..cstart[i+1]     children of internal[i] (indices into child[])
//   child[j]                   child node id
//   leaf_col[node]             counts column of a leaf, -1 for internal
//   slot[node]                 scratch slot of an internal node
struct TreePlan {
    int n_nodes;
    int n_internal;
    int n_leaves;
    int root;
    int n_slots;
    int max_children;
    const int32_t* internal;
    const int32_t* cstart;
    const int32_t* child;
    const int32_t* leaf_col;
    const int32_t* slot;
};

constexpr int kMaxNodes = 512;

}  // namespace cafe

// Launch wrappers implemented in the .cu files (host side).
namespace cafe {

cudaError_t launch_matrix_build(const MatrixJob* d_jobs, int n_jobs, int max_size, int sm_count, cudaStream_t s);

// ---- distinct count patterns per subtree (k_patterns.cu) ----
constexpr int kMaxGroups = 16;
struct PatBuildArgs {
    TreePlan plan;
    const int32_t* counts;       // [F][n_leaves]
    const int64_t* perm;         // [F] family of each item (group order)
    const int32_t* node_ii;      // [n_nodes] post-order index of an internal node, -1 for leaves
    int64_t F;
    int n_groups;
    const int64_t* group_first;  // [n_groups + 1] first item of a group; then F
    const int64_t* flag_off;     // [n_groups] a group's first entry in the flags of launch_pat_counts
    const int32_t* group_max;    // [n_groups] its largest count
    int32_t* rep;                // [n_internal][F] the item that represents an item's key at a node
    int32_t* num;                // [n_internal][F] representatives before an item
    int32_t* base;               // [n_internal][n_groups + 1] num at each group's first item; then the total
};
// nodes: post-order indices of one level; the table holds n_nodes x slots
// (a power of two, at least 2 F) entries, all -1
cudaError_t launch_pat_insert(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, int32_t* table, int64_t slots,
                              cudaStream_t s);
// flags: [leaf][group_max + 1] per group, zeroed in; 1 where the count occurs
cudaError_t launch_pat_counts(const PatBuildArgs& a, uint8_t* flags, cudaStream_t s);
// nodes: post-order indices of the deduplicated nodes
cudaError_t launch_pat_number(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, cudaStream_t s);
// child_off [n_groups][n_internal]: first child index of a (group, node) in
// `child`; nodes may include the root
cudaError_t launch_pat_write(const PatBuildArgs& a, const int32_t* d_nodes, int n_nodes, const int64_t* d_child_off,
                             int32_t* d_child, cudaStream_t s);

// ---- FP64 pruning over distinct rows (k_pat64.cu) ----
// One node of one group. An internal node's `rows` distinct vectors become
// factor rows F[row][s] = sum_j M[s][j] L[row][j] (s < s_cnt) in the
// combination's table; a leaf's rows are the factors of counts 0.. (the last
// row stands for all larger counts; only counts that occur are filled in);
// the root's rows are the group's families.
struct Pat64Node {
    int64_t tab;                 // first element of the node's factor rows in a combination's table
    int64_t cidx;                // first of its rows' child indices; a leaf: of its counts in `leaf_counts`
    int64_t perm0;               // root: first item of the group
    int32_t unit0, n_units;      // its work units in a combination's list
    int32_t rows;
    int32_t n_list;              // a leaf's counts
    int32_t node, nch;           // tree node, its children (0: a leaf)
    int32_t S;                   // the group's states 0..S
    int32_t s_cnt, pitch;        // factor entries per row, row pitch
    int32_t s_tiles;             // state tiles of a row tile
    int32_t erow0;               // first entry of its rows in the exponent table
    int32_t child0;              // its children in cdesc
    int32_t root;                // the group's root (index of its Pat64Node)
    int32_t R;                   // root rows: root sizes 1..R
};
struct Pat64Args {
    TreePlan plan;
    const Pat64Node* nodes;      // [n_desc] by height, so children come first
    const int32_t* cdesc;        // per node and child: the child's Pat64Node
    int n_desc;
    int units;                   // units of one combination
    int s_run;                   // state tiles of a unit
    int n_bufs;                  // vector buffers of a CTA
    int64_t buf_doubles;
    // max-product (ctab not null): the argmax of every factor, laid out like
    // table; FP32 log2 of each matrix [S + 1][lm_pitch] and its chunk maxima
    // (launch_log2_rows); the families' root values and states
    int32_t* ctab;
    const float* const* lmats;   // [K][n_nodes], null at leaves and the root
    int lm_pitch;
    int64_t F;
    double* root_max;            // [K][F]
    int32_t* root_arg;           // [K][F]
    int32_t* n_failed;           // families with root value 0
    double* root_out;            // not null: every family's root vector (root sizes 1..R) instead of
                                 // the root weighting, [F][R]
    const int32_t* active;       // [n_active] combined (candidate, category) indices
    int n_active;
    int group;                   // combinations interleaved unit by unit
    int n_slots;                 // combinations whose tables exist at a time
    int64_t slot_doubles, slot_rows;
    double* table;               // [n_slots][slot_doubles]
    int32_t* expo;               // [n_slots][slot_rows] power-of-two exponents of the rows
    int32_t* done;               // [n_active][n_desc] finished units, zeroed
    unsigned long long* next;    // unit counter, zeroed
    int32_t* status;             // nonzero when a bounded wait gave up
    const int32_t* child;        // child indices (launch_pat_write)
    const int32_t* leaf_counts;  // the counts that occur at a leaf
    const int64_t* perm;
    const double* const* mats;   // [K][n_nodes]
    int ld_mat;
    const double* prior;
    int n_prior;
    const double* err;
    int err_rows, err_ndev;
    const int32_t* fam_R;
    int scaled, model;
    double* out;                 // [F][K]
    int K;
    const double* cat_probs;
};
constexpr int kPat64RootRows = 8;   // families of a root unit
constexpr int kPat64Rows = 8;       // rows of any other
constexpr int kPat64States = 16;    // states of a state tile
// lp: pitch of the longest vectors in shared memory (whole 32-state chunks,
// plus 2)
int pat64_bufs(int lp, int max_R, bool max_product = false);
int64_t pat64_buf_doubles(int lp, int max_R, bool max_product = false);
cudaError_t pat64_init();
cudaError_t launch_pat64(const Pat64Args& a, int n_ctas, cudaStream_t s);
int pat64_ctas_per_sm(size_t smem, bool max_product = false);

struct Prune64Args {
    TreePlan plan;
    const PruneTile* tiles;
    int n_tiles;
    const int32_t* counts;       // [F][n_leaves]
    const int64_t* perm;         // family index of each tile slot
    const double* const* mats;   // [K][n_nodes] FP64 matrix per (category, node)
    int ld_mat;                  // row stride of every FP64 matrix (= matrix size)
    const double* prior;         // [n_prior]
    int n_prior;
    const double* err;           // [err_rows][err_ndev] or null
    int err_rows;
    int err_ndev;
    const int32_t* fam_R;        // per-family root bound, or null (tile R)
    double* scratch;             // n_ctas * per_cta doubles
    int64_t scratch_per_cta;
    int scaled;                  // per-node power-of-two rescale
    int model;                   // 0 base, 1 gamma
    double* out;                 // [F][K]: base lnl, gamma category value
    int K;                       // categories (all candidates' categories of a batch)
    const double* cat_probs;     // [K]
    int tile_families;           // families per tile (<= 32)
    int W;                       // max vector length over tiles (S + 1 or R)
    const int32_t* n_tiles_dev;  // optional: tile count read from device memory
    double* root_out;            // optional (unscaled runs): root vector of every family,
                                 // root_out[f * root_ld + j] = L(root size root_lo + j); no reduction
    int root_ld;
};

cudaError_t launch_prune64(const Prune64Args& a, int n_ctas, cudaStream_t s);

struct FinishArgs {
    int64_t F;
    int K;                       // categories per candidate (1 for the base model)
    int n_cand;                  // candidates scored together (>= 1)
    int model;
    int scaled;
    const double* cat;           // [F][n_cand][K]: gamma terms (linear if !scaled, log if scaled); base: lnl
    double* family_lnl;          // [n_cand][F] out, or null
    double* total;               // [n_cand] out, or null
    int32_t* n_failed;           // [n_cand] out
    double* part_sum;            // [n_cand][2 * finish_parts(F)] workspace
    int32_t* part_cnt;           // [n_cand][2 * finish_parts(F)] workspace
    const int32_t* status;       // optional: nonzero -> total = NaN
};

int finish_parts(int64_t F);
cudaError_t launch_finish(const FinishArgs& a, cudaStream_t s);

// ---- tensor-core (TF32x3) path ----
// Conversion of one cached FP64 matrix into the tensor-core operands.
struct ConvertJob {
    const double* src;   // FP64 row-major, leading dimension `ld`
    int ld;
    int mat;             // index into the request's converted arrays
    int what;            // 1: the TF32 hi/lo operands (an internal child's branch), 2: the
                         // FP32 transpose (a leaf's branch); both where a matrix serves both
};

struct TcBuffers {
    float* hi;           // [n_mat][Wm][Wm] TF32 hi part, row-major M[s][c]
    float* lo;           // [n_mat][Wm][Wm] TF32 lo part
    float* tr;           // [n_mat][Wm][Wm] FP32 transpose: tr[c][s] = M[s][c] (leaf factors); with an
                         // error model, the leaf factor of an observed count c: sum over deviations d of
                         // w_d(c) M[s][c + d] (columns 0 .. Wm - 1, zero weights skipped), summed in FP32
                         // in deviation order
    int Wm;
    const double* err;   // [err_rows][err_ndev] error model, or null
    int err_rows, err_ndev;
};
constexpr int kMaxErrHalf = 8;   // deviations up to +-8 fold into the transposed leaf rows

cudaError_t launch_convert_tc(const ConvertJob* d_jobs, int n_jobs, TcBuffers b, cudaStream_t s);

// ---- tensor-core pruning over distinct rows (k_pat_tc.cu) ----
struct PatTcNode {               // an internal node of the bin, by height; the root last
    int64_t cidx, perm0;         // first child index of its rows; root: first item
    int32_t unit0, n_units;      // first unit in its level, units
    int32_t rows, row0;          // rows (root: families), first row in a combination's table (a multiple of 32)
    int32_t node, nch;           // tree node, children (1 or 2)
    int32_t child[2], child_node[2];   // the children's PatTcNode (-1: a leaf) and tree nodes
};
// The units of one level of combinations q0 .. q0 + nq - 1, the combinations
// interleaved.
struct PatTcSeg {
    long long unit0;             // first unit in the launch's order
    int32_t q0, nq;
    int32_t node0, node1;        // the level's nodes
};
struct PatTcArgs {
    const PatTcNode* nodes;
    const PatTcSeg* segs;
    int n_desc, n_segs;
    long long total_units;
    const int32_t* active;       // combined (candidate, category) indices
    int n_slots;                 // combinations whose tables exist at a time
    int64_t slot_rows;           // table rows per combination
    float* table;                // [n_slots][slot_rows][W] factor rows
    int4* meta;                  // [n_slots][slot_rows] exponent, flags, error bound
    int32_t* done;               // [n_active][n_desc] finished units, zeroed
    unsigned long long* next;    // unit counter, zeroed
    int32_t* status;             // nonzero when a bounded wait gave up
    int32_t* any_flag;           // set when a family is left to FP64
    const int32_t* child;        // child indices (launch_pat_write)
    const int64_t* perm;
    const int32_t* mat_index;    // [K][n_nodes] converted-matrix index; bit 30: the key is saturated
    int n_nodes;
    int W, Wm;                   // bin width; pitch of the converted matrices
    int Ns, n_share;             // states of a unit, units along the states
    int tmem_cols;
    const int32_t* item_R;       // [F] root bound of each item
    const float* mat_tr;         // [n_mat][Wm][Wm] FP32 transposed matrices (row c = column c of M)
    const double* prior;
    int n_prior;
    const double* err;
    int err_rows, err_ndev;
    double* out;                 // [F][K] natural log of each category term
    float* out_err;              // [F][K] bound on its relative error from FP32 range loss
    int K, model;                // model 0 base (a zero family is -inf), 1 gamma (a zero family is NaN: failed)
    const double* cat_probs;
    int32_t* flags;              // [F] set when a family must be recomputed in FP64
    uint8_t* term_flags;         // [F][K] set with it for the category term that needs the recompute
    int debug_wait_limit;        // > 0: the wait for a unit's GEMM gives up after this many polls minus one
};
int pat_tc_states(int W);
cudaError_t pat_tc_init();
int pat_tc_ctas_per_sm(int W);
// mat: the TF32 hi and lo matrices [2][n_mat Wm][Wm] in boxes of 32 columns x
// Ns rows x both; vst, vst32: the factor tables [n_slots slot_rows][W] in boxes
// of 32 columns x 128 or 32 rows (all 128-byte swizzled)
struct PatTcMaps {
    CUtensorMap mat, vst, vst32;
};
cudaError_t launch_pat_tc(const PatTcMaps& m, const PatTcArgs& a, int n_ctas, cudaStream_t s);

// ---- device-sampled p-value simulations (k_pvalue.cu) ----
struct SimDrawArgs {
    const double* cdf;           // [n_nodes][n_ps][S] cumulative weights of each (node, parent size) row
    const int32_t* prefix;       // [n_nodes] prefix order
    const int32_t* parent;       // [n_nodes], -1 at the root
    const int32_t* leaf_col;     // [n_nodes] counts column of a leaf, -1 for internal nodes
    int n_nodes, n_leaves, root, n_ps, S, n_sim;
    int64_t n_families;          // R x n_sim; family fi has root size fi / n_sim + 1
    uint64_t key;                // sim_seed_key(seed)
    const uint2* words;          // the reference's stream: two words a draw, and each family's
    const int64_t* starts;       // first draw; null: draws by (family, node)
    int32_t* sizes;              // [n_families][n_nodes] scratch
    int32_t* counts;             // [n_families][n_leaves] out: leaf counts
    int R;
    int32_t* keys;               // [n_families] out: state bound x R + root index
    int32_t* hist;               // [(S + 1) x R] zeroed in, families per key out
};
struct SimPlanArgs {
    const int32_t* hist;
    int S, R;
    int32_t* cursor;             // [n_keys] out: first family slot of each key (the scatter's cursor)
    PruneTile* tiles;            // [max_tiles] out: 32-family tiles of equal (root size, bound)
    int64_t max_tiles;
    int32_t* n_tiles;            // [1] out
    int64_t* bound_first;        // [S + 2] out: first family slot of each state bound; then the families
};
// Root values of the simulated families i0 <= i < i1 (in slot order) from the
// factor rows of the root's grandchildren (k_pat64).
struct SimRootArgs {
    TreePlan plan;
    const int32_t* node_ii;      // [n_nodes] post-order index of an internal node, -1 for leaves
    const int32_t* keys;         // state bound x R + root index
    int R;
    const int32_t* counts;       // [n_families][n_leaves]
    const int64_t* perm;
    int64_t i0, i1, F;
    int n_groups;
    const int32_t *rep, *num, *base;   // PatBuildArgs
    const int64_t* tab;          // [n_groups][n_nodes] a node's factor rows in `table`, pitch (bound + 2) & ~1
    const double* table;
    int leaf_pitch;              // (a leaf's rows, by count, serve every group)
    const double* const* mats;
    int ld_mat;
    double* out;                 // [n_families]
};
struct PvalueSearchArgs {
    const int32_t* counts;       // [F][n_leaves] observed families
    int64_t F;
    int n_leaves;
    const double* obs;           // [F][R] observed root values (root sizes 1..R)
    const double* sorted;        // [R][n_sim] sorted simulated values
    int R, n_sim;
    double* out;                 // [F] p-values
};
constexpr int kSortRowsMaxP = 16384;   // simulations per root size the device sort takes
uint64_t sim_seed_key(uint32_t seed);
cudaError_t pvalue_kernels_init();
// normalised: weights over their sum, as std::discrete_distribution keeps them
cudaError_t launch_cdf_build(const double* const* mats, int n_nodes, int msize, int S, int n_ps, bool normalised,
                             double* cdf, cudaStream_t s);
// Where every family's draws start in one std::mt19937's stream (k_pvalue.cu).
struct SimStreamArgs {
    const double* cdf;           // normalised rows
    const int32_t* prefix;       // as in SimDrawArgs
    const int32_t* parent;
    const int32_t* leaf_col;
    const int32_t* node_ii;      // [n_nodes] index of an internal node, -1 for leaves
    int n_nodes, n_internal, root, n_ps, S, n_sim;
    const uint2* words;          // [R n_sim (n_nodes - 1)]
    uint16_t* len;               // [(n_sim - 1) (n_nodes - 1) + 1] scratch
    int64_t* starts;             // [R n_sim + 1] out; the first is set
    int32_t* state;              // [4] root sizes done, first one that is not regular (INT_MAX), CTAs
                                 // done, whether the next one needs every start
};
constexpr int kMtWords = 624;
// the next n words of the stream whose state [kMtWords] is kept on the device
// (n a multiple of kMtWords but in the last call); first: seeded here
cudaError_t launch_mt_words(bool first, uint32_t seed, uint32_t* state, int64_t n, uint32_t* out, cudaStream_t s);
cudaError_t launch_sim_starts(const SimStreamArgs& a, int r0, int r1, cudaStream_t s);      // root sizes up to r1, of
                                                                                            // which r0 may be open
cudaError_t launch_sim_draw(const SimDrawArgs& a, cudaStream_t s);
cudaError_t launch_sim_plan(const SimPlanArgs& a, cudaStream_t s);
cudaError_t launch_sim_root(const SimRootArgs& a, cudaStream_t s);
cudaError_t launch_sim_scatter(const int32_t* keys, int64_t n, int32_t* cursor, int64_t* perm, cudaStream_t s);
cudaError_t launch_sort_rows(double* v, int rows, int n, cudaStream_t s);
cudaError_t launch_pvalue_search(const PvalueSearchArgs& a, cudaStream_t s);

// Families whose tensor-core result may have lost accuracy to FP32's range:
// for every (family, candidate), the category terms' range-error bounds
// weighted by the terms' shares of the family likelihood; over
// tau x |lnL| the family is flagged for the FP64 recompute.
struct RangeFlagArgs {
    const double* cat;           // [F][K] natural log of each category term
    const float* err;            // [F][K] relative bound of each term
    int64_t F;
    int K;                       // combined (candidate, category) indices
    int KC;                      // categories per candidate
    double tau;
    int32_t* flags;              // [F]
    uint8_t* term_flags;         // [F][K]: the terms of a flagged family whose share of the bound is over
                                 // tau / (2 KC), which the FP64 pass recomputes (the rest stay under tau / 2)
    int32_t* any_flag;           // set to 1 when a family is flagged
};
cudaError_t launch_range_flags(const RangeFlagArgs& a, cudaStream_t s);

// ---- FP64 recompute of flagged category terms (k_terms64.cu) ----
struct TermTile {
    int32_t first;               // a chunk of 32 families (perm order) of a bin
    uint32_t mask;               // the tile's families among them, at most four
    int32_t k, W;                // category, bin width
};
struct TermTileArgs {
    const int32_t* flags;        // [F]
    const uint8_t* term_flags;   // [F][K]
    int K;                       // combined (candidate, category) indices
    const int64_t* perm;         // [F] bin order
    int n_bins;
    int bin_width[16];
    int64_t bin_first[16];
    int64_t bin_count[16];
    const int32_t* cats;         // [n_cats] category indices to recompute
    int n_cats;
    TermTile* tiles;             // [term_tiles_max]
    int32_t* out_counts;         // [2] flagged families, tiles; zeroed in
    const int32_t* any_flag;     // zero: no family is flagged
};
struct TermArgs {
    TreePlan plan;
    const TermTile* tiles;
    const int32_t* n_tiles;
    const int32_t* counts;
    const int64_t* perm;
    const double* const* mats;   // [K][n_nodes]
    int ld_mat;
    int W;                       // widest bin
    const double* prior;
    int n_prior;
    const double* err;
    int err_rows, err_ndev;
    const int32_t* fam_R;
    int model;
    double* out;                 // [F][K]
    int K;
    const double* cat_probs;
};
int64_t term_tiles_max(int64_t F, int n_bins, int n_cats);
cudaError_t terms64_init();
cudaError_t launch_term_tiles(const TermTileArgs& a, int sm_count, cudaStream_t s);
cudaError_t launch_terms64(const TermArgs& a, int sm_count, cudaStream_t s);

// ---- Pupko joint reconstruction (k_reconstruct.cu) ----
// One CTA walks 32-family tiles of one category up the tree; node L
// vectors (S + 1 states) live in per-CTA scratch, the argmax tables C in
// per-CTA int32 scratch; the backtrack writes every node's state.
struct PupkoArgs {
    TreePlan plan;
    const PruneTile* tiles;      // first family, count (<= 32), category k
    int n_tiles;
    const int32_t* counts;       // [F][n_leaves]
    int64_t F;
    const double* const* mats;   // [K][n_nodes] FP64 matrix per (category, node)
    const float* const* lmats;   // [K][n_nodes] transposed log2 of the internal non-root nodes' matrices,
                                 // (S + 1) x (S + 1) (launch_log2_matrices), null elsewhere
    int ld_mat;                  // matrix side (>= S + 1)
    const double* prior;         // prior[j] = P(root size j)
    int n_prior;
    int S;                       // max_family_size: states 0..S
    int root_len;                // min(S, R) + 1: root sizes 1..root_len - 1
    double* scratch;             // n_ctas * scratch_per_cta doubles
    int64_t scratch_per_cta;     // pupko_scratch_doubles()
    int32_t* cscratch;           // n_ctas * c_per_cta
    int64_t c_per_cta;           // pupko_c_entries()
    int32_t* state;              // [K][F][n_nodes] out
    double* root_max;            // [K][F] out
    int32_t* n_failed;           // [1] out: (category, family) pairs with root max 0
    int exhaustive;              // 1: exact FP64 scan of every child state
};
cudaError_t launch_pupko(const PupkoArgs& a, int n_ctas, cudaStream_t s);
cudaError_t launch_log2_matrices(const double* const* src, float* const* dst, int n_mats, int n, int ld,
                                 cudaStream_t s);
// log2 of each matrix's first n x n block, row-major with pitch `pitch` (-inf
// past n), then the largest of every 32 columns [n][pitch / 32]
cudaError_t launch_log2_rows(const double* const* src, float* const* dst, int n_mats, int n, int ld, int pitch,
                             cudaStream_t s);
// Every family's states from the root's (parents before children): a node's row
// among its distinct patterns follows from its parent's.
struct BacktrackArgs {
    TreePlan plan;
    const int32_t* node_ii;      // [n_nodes] post-order index of an internal node, -1 for leaves
    const int64_t* child_off;    // [n_internal] first child index of a node
    const int32_t* child;        // child indices (a leaf's: the count)
    const int64_t* ctab_off;     // [n_internal] first entry of a node's argmax table
    const int32_t* pitch;        // [n_internal] its row pitch
    const int32_t* ctab;         // of category k0, the next ones ctab_stride further
    int64_t ctab_stride;
    const int32_t* root_arg;     // [K][F]
    const int32_t* status;       // nonzero: the tables are incomplete
    int64_t F;
    int64_t f0, nf;              // families f0 .. f0 + nf - 1, whose patterns these are
    int k0, n_k;                 // categories k0 .. k0 + n_k - 1
    int32_t* row;                // [n_k][nf][n_internal] scratch
    int32_t* state;              // [K][F][n_nodes] out
};
cudaError_t launch_backtrack(const BacktrackArgs& a, cudaStream_t s);
size_t pupko_scratch_doubles(const TreePlan& P, int S);
size_t pupko_c_entries(const TreePlan& P, int S);
cudaError_t launch_recon_counts(const int32_t* state, int64_t F, int n_nodes, int K, const double* cat_probs,
                                int gamma, const int32_t* leaf_col, double* mean, int32_t* node_count,
                                cudaStream_t s);

struct BranchProbArgs {
    const int32_t* parent;       // [n_nodes], -1 at the root
    int n_nodes;
    int64_t F;
    const int32_t* node_count;   // [F][n_nodes]
    const double* const* mats;   // [n_nodes] matrix of the branch above each node
    int ld_mat;
    int S;                       // child sizes 0..S-1 are summed
    double* out;                 // [F][n_nodes], NaN at the root
    int32_t* n_bad;              // [1] counts outside the matrices
};
cudaError_t launch_branch_prob(const BranchProbArgs& a, cudaStream_t s);

}  // namespace cafe
