"""FP64 scores over distinct subtree patterns (k_patterns, k_pat64): row,
state and chunk counts at the edges of a unit (8 rows, 16-state tiles,
32-column chunks), repeated and distinct rows, polytomies, a unary node, an
error model, and batches. Against the FP64 oracle; tolerance 1e-12 relative
per family (the oracle's own sums round differently, by a few 1e-16 per node
and at most a few dozen nodes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINARY = "((A:3.2,B:3.2):4.5,((C:2.5,D:2.5):1.25,E:3.75):3.95);"
POLY = "((A:3.2,B:3.2,C:3.2):4.5,(D:2.5,(E:1.5):1.0,F:2.5):5.2,G:7.7);"


@pytest.fixture(scope="module")
def ctx():
    from cafe5_gb300.engine import Context
    c = Context()
    yield c
    c.close()


def _oracle():
    import os
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
    import oracle
    return oracle


def _counts(rng, F, n_leaves, hi, distinct):
    """`distinct` different rows among F."""
    base = rng.integers(0, hi + 1, (max(distinct, 1), n_leaves))
    base[:, 0] = np.maximum(base[:, 0], 1)
    return np.ascontiguousarray(base[rng.integers(0, len(base), F)], dtype=np.int32)


@pytest.mark.parametrize("newick", [BINARY, POLY], ids=["binary", "polytomy"])
@pytest.mark.parametrize("F,distinct,hi,S,R", [
    (1, 1, 3, 15, 10),        # one row, one tile
    (7, 7, 5, 16, 16),        # a tile and one state over
    (8, 3, 5, 30, 31),        # root sizes past the states
    (9, 9, 9, 31, 20),        # one row over; a whole chunk
    (65, 40, 12, 32, 40),     # a chunk and one column over
    (300, 40, 20, 130, 100),  # chunks that leave every partial sum unchanged
    (40, 40, 120, 170, 150),  # large counts at the reference's bounds
])
@pytest.mark.parametrize("eps", [0.0, 0.07])
def test_fp64_ref_rows(ctx, newick, F, distinct, hi, S, R, eps):
    oracle = _oracle()
    from cafe5_gb300.inputs import ErrorModel, RootPrior
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick(newick)
    rng = np.random.default_rng([F, distinct, S])
    c = _counts(rng, F, len(tree.leaves), min(hi, S), distinct)
    prior = RootPrior.uniform(R).vector()
    em = ErrorModel.symmetric(eps, int(c.max())) if eps else None
    tid = ctx.upload_tree(tree)
    sid = ctx.upload_families(tid, c)
    ctx.set_prior(prior)
    ctx.set_error_model(em.table() if em else None)
    ta = oracle.TreeArrays.from_tree(tree)
    lams = [0.004, 0.013]
    got = ctx.score_batch(tid, sid, [dict(lambdas=[l]) for l in lams], S=S, R=R, use_error_model=em is not None)
    for l, r in zip(lams, got):
        _, fam, _ = oracle.score(ta, c, [l], prior=prior, S=S, R=R, err_rows=em.table() if em else None)
        ok = np.isfinite(fam)
        assert np.array_equal(ok, np.isfinite(r.family_lnl))
        assert np.all(np.abs(r.family_lnl[ok] - fam[ok]) <= 1e-12 * np.maximum(1.0, np.abs(fam[ok])))
        # the same bits alone, and for equal families
        assert np.array_equal(r.family_lnl, ctx.score(tid, sid, [l], S=S, R=R, use_error_model=em is not None).family_lnl)
    _, inv = np.unique(c, axis=0, return_inverse=True)
    for g in range(inv.max() + 1):
        assert len(set(got[0].family_lnl[inv.reshape(-1) == g])) == 1
    ctx.free_families(sid)
    ctx.set_error_model(None)


def test_fp64_binned_tables_are_reused_across_combinations(ctx):
    """More (candidate, category) combinations than factor tables: every table
    is taken over by later ones; each candidate keeps the bits it has alone."""
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.synth import workload
    w = workload(1, n_families=6000, seed=9)
    tid = ctx.upload_tree(w.tree)
    sid = ctx.upload_families(tid, w.families.counts)
    ctx.set_prior(RootPrior.uniform(150).vector())
    cands = [dict(lambdas=[0.002 * (1 + 0.01 * b)], multipliers=w.multipliers, cat_probs=w.cat_probs) for b in range(24)]
    got = ctx.score_batch(tid, sid, cands, model=1, precision="fp64_binned")
    for b in (0, 11, 23):
        alone = ctx.score(tid, sid, cands[b]["lambdas"], model=1, precision="fp64_binned", multipliers=w.multipliers,
                          cat_probs=w.cat_probs)
        assert np.array_equal(alone.family_lnl, got[b].family_lnl) and alone.total == got[b].total
    ctx.free_families(sid)


@pytest.mark.parametrize("newick", [BINARY, POLY, "(A:1.0,B:2.0);"], ids=["binary", "polytomy", "root only"])
@pytest.mark.parametrize("F,distinct,hi,S,R", [
    (1, 1, 3, 15, 10),
    (7, 7, 5, 16, 40),        # root sizes past the states
    (9, 9, 9, 30, 20),        # 31 states
    (33, 20, 12, 31, 31),     # a whole chunk
    (65, 40, 12, 32, 5),      # a chunk and one column over
    (300, 120, 60, 130, 100),
    (17, 17, 200, 511, 300),  # sixteen chunks
])
@pytest.mark.parametrize("lam", [0.01, 1e-9])     # (the second: most products are subnormal or zero)
def test_reconstruction_rows(ctx, newick, F, distinct, hi, S, R, lam):
    """Joint reconstruction over distinct rows against the walk that forms every
    product in FP64: the same bits and states."""
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick(newick)
    c = _counts(np.random.default_rng([F, S]), F, len(tree.leaves), min(hi, S), distinct)
    tid = ctx.upload_tree(tree)
    sid = ctx.upload_families(tid, c)
    ctx.set_prior(RootPrior.uniform(R).vector())
    kw = dict(S=S, R=R, model=1, multipliers=[0.3, 0.9, 2.0], cat_probs=[0.2, 0.5, 0.3])
    a, b = ctx.reconstruct(tid, sid, [lam], **kw), ctx.reconstruct(tid, sid, [lam], exhaustive=True, **kw)
    for x, y in ((a.category_state, b.category_state), (a.node_count, b.node_count), (a.node_mean, b.node_mean),
                 (a.root_max, b.root_max)):
        assert np.array_equal(x, y)
    assert a.n_failed == b.n_failed
    ctx.free_families(sid)


@pytest.mark.parametrize("newick", [BINARY, POLY, "(A:1.0,B:2.0);"], ids=["binary", "polytomy", "root only"])
@pytest.mark.parametrize("n_sim,S,R,lam,seed", [
    (1, 2, 1, 0.05, 1),          # a draw between two sizes
    (31, 16, 40, 0.02, 0),       # root sizes past the states
    (33, 60, 20, 0.05, 7),       # most families die out somewhere: draws are skipped
    (3201, 40, 3, 0.03, 2**32 - 1),   # more families than one segment of the chain of starts holds
    (300, 130, 90, 0.004, 10),   # several state bounds
])
def test_pvalue_rows_and_stream(ctx, newick, n_sim, S, R, lam, seed):
    """The reference's stream followed on the device, and the simulated families
    pruned over distinct rows: the conditional distributions against the
    oracle's, 1e-10 relative (two orders of summation, as for the p-values'
    other tests), zeros in the same places."""
    oracle = _oracle()
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick(newick)
    c = _counts(np.random.default_rng(5), 3, len(tree.leaves), min(S, 12), 3)
    tid = ctx.upload_tree(tree)
    sid = ctx.upload_families(tid, c)
    got = ctx.pvalues(tid, sid, [lam], S=S, R=R, n_simulations=n_sim, seed=seed)
    _, cd, rv = oracle.pvalues(oracle.TreeArrays.from_tree(tree), c, [lam], S=S, R=R, n_sim=n_sim, seed=seed)
    for x, y in ((got["conditional"], cd), (got["root_likelihood"], rv)):
        assert np.array_equal(x > 0, y > 0)
        assert np.all(np.abs(x - y) <= 1e-10 * y)
    ctx.free_families(sid)


@pytest.mark.parametrize("hi", [10, 40, 120, 420])           # bins of 64, 96, 192 and 512 states
@pytest.mark.parametrize("eps", [0.0, 0.07])
def test_flagged_terms(ctx, hi, eps):
    """The FP64 recompute of flagged terms (k_term_tiles, k_terms64): nearly
    diagonal matrices and unequal counts put the FP32 range bound over budget.
    With one category a flagged family's result is its fp64_binned one, bit for
    bit; the others are within 1e-6."""
    from cafe5_gb300.inputs import ErrorModel, RootPrior
    from cafe5_gb300.synth import workload
    w = workload(1, n_families=10, seed=3)
    tid = ctx.upload_tree(w.tree)
    flagged = 0
    for F in (1, 4, 5, 33, 300):            # one tile; full; one over; a second chunk; many
        rng = np.random.default_rng([F, hi])
        c = rng.integers(max(hi - hi // 4, 0), hi + 1, (F, len(w.tree.leaves)), dtype=np.int32)
        c[:, rng.integers(0, c.shape[1])] = 1
        em = ErrorModel.symmetric(eps, int(c.max())) if eps else None
        ctx.set_prior(RootPrior.uniform(int(c.max() * 1.25) + 1).vector())
        ctx.set_error_model(em.table() if em else None)
        sid = ctx.upload_families(tid, c)
        kw = dict(use_error_model=em is not None)
        b, m = (ctx.score(tid, sid, [1e-5], precision=p, **kw) for p in ("fp64_binned", "mixed_tf32x3"))
        flagged += m.n_fallback
        assert np.array_equal(np.isfinite(b.family_lnl), np.isfinite(m.family_lnl))
        ok = np.isfinite(b.family_lnl)
        assert np.all(np.abs(m.family_lnl[ok] - b.family_lnl[ok]) <= 1e-6 * np.abs(b.family_lnl[ok]))
        assert np.sum(m.family_lnl[ok] == b.family_lnl[ok]) >= m.n_fallback - np.sum(~ok)
        ctx.free_families(sid)
    ctx.set_error_model(None)
    assert flagged > 0


@pytest.mark.parametrize("hi", [8, 30, 45, 100, 300])        # bins of 32, 64, 96, 128 / 192 and 512 states
@pytest.mark.parametrize("newick", [None, "((A:3.2,B:3.2):4.5,((C:2.5,(D:1.5):1.0):1.25,E:3.75):3.95);"],
                         ids=["48 taxa", "one-child node"])
def test_tensor_core_rows(ctx, newick, hi):
    """k_pat_tc at the edges of its row tiles (128 rows, stored 32 at a time, the
    root's last tile down to one family) with many combinations in flight: the
    same bits on every call, and within 1e-6 of fp64_binned."""
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.synth import workload
    from cafe5_gb300.tree import parse_newick
    w = workload(3, n_families=10, seed=3)
    tree = parse_newick(newick) if newick else w.tree
    tid = ctx.upload_tree(tree)
    cands = [dict(lambdas=[0.002 * (1 + 0.05 * b)], multipliers=[0.3, 0.7, 1.1, 1.9], cat_probs=[0.25] * 4)
             for b in range(24)]
    for F in (1, 33, 97, 128, 131, 273):
        rng = np.random.default_rng([F, hi])
        c = _counts(rng, F, len(tree.leaves), hi, F)
        c = np.ascontiguousarray(np.maximum(c, hi // 2))
        ctx.set_prior(RootPrior.uniform(int(c.max() * 1.25) + 1).vector())
        sid = ctx.upload_families(tid, c)
        ref = ctx.score_batch(tid, sid, cands, model=1, precision="fp64_binned")
        first = None
        for _ in range(3):
            got = ctx.score_batch(tid, sid, cands, model=1, precision="mixed_tf32x3")
            for a, b in zip(got, ref):
                x, y = a.family_lnl, b.family_lnl
                ok = np.isfinite(y)             # (a saturated candidate is NaN in both)
                assert a.status == b.status and np.array_equal(np.isfinite(x), ok)
                assert np.all(np.abs(x[ok] - y[ok]) <= 1e-6 * np.abs(y[ok]))
            if first:
                assert all(np.array_equal(a.family_lnl, b.family_lnl, equal_nan=True) for a, b in zip(got, first))
            first = got
        ctx.free_families(sid)


@pytest.mark.parametrize("size", [1, 2, 3, 8, 9, 10, 31, 32, 33, 63, 64, 65, 66, 72, 97, 129, 171, 258])
def test_matrix_rows(ctx, size):
    """k_matrix_build at the edges of its warps (32 row pairs) and tiles (8
    steps): odd and even sides, rows that underflow at their left end, the
    rescaled ones, saturated keys. 1e-12 relative to the oracle where it is at
    least 1e-280, as for the larger builds."""
    oracle = _oracle()
    lams, ts = [1e-6, 0.0025, 0.011, 0.6], [0.001, 0.5, 14.25, 40.0]
    ctx.matrices_build(lams, ts, size)
    for lam in lams:
        for t in ts:
            ours, ref = ctx.matrix_get(lam, t, size), oracle.fill_matrix(lam, t, size)
            mask = ref >= 1e-280
            assert np.all(np.abs(ours[mask] - ref[mask]) <= 1e-12 * ref[mask]), (lam, t)
            assert np.all(ours[~mask] <= 1e-270)
