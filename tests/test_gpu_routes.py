"""Routes that ordinary sizes do not take, against the oracle or the route that
they do: vectors past a CTA's shared memory, one-child nodes, p-values whose
draws stay on the host, and the tile walk's ranked maxima."""
import numpy as np
import pytest

from cafe5_gb300 import _lib

pytestmark = pytest.mark.gpu

BINARY = "((A:3.2,B:3.2):4.5,((C:2.5,D:2.5):1.25,E:3.75):3.95);"


@pytest.fixture(scope="module")
def ctx():
    from cafe5_gb300.engine import Context
    c = Context()
    yield c
    c.close()


def _upload(ctx, newick, counts, n_prior):
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick(newick)
    tid = ctx.upload_tree(tree)
    ctx.set_prior(RootPrior.uniform(n_prior).vector())
    return tree, tid, ctx.upload_families(tid, np.ascontiguousarray(counts, np.int32))


def test_fp64_vectors_past_shared_memory(ctx):
    """Past 3,167 states eight vectors do not fit a CTA and the tile walk takes
    them. The states between 3,100 and 3,200 add nothing at these counts (below
    1e-300 of the sums), so both bounds give the same likelihoods but for the
    rounding of the sums: 1e-13 relative."""
    rng = np.random.default_rng(2)
    tree, tid, sid = _upload(ctx, BINARY, rng.integers(1, 25, (37, 5)), 60)
    rows, tiles = (ctx.score(tid, sid, [0.01], S=S, R=60).family_lnl for S in (3100, 3200))
    assert np.all(np.isfinite(rows))
    assert np.all(np.abs(rows - tiles) <= 1e-13 * np.abs(rows))


def test_reconstruction_vectors_past_shared_memory(ctx):
    """The same for max-products, whose vectors take twice the memory: k_pupko's
    ranked maxima at 2,300 states, k_pat64's at 1,200; the extra states are never
    the largest, so states and root values are equal."""
    rng = np.random.default_rng(3)
    tree, tid, sid = _upload(ctx, BINARY, rng.integers(0, 25, (37, 5)), 60)
    rows, tiles = (ctx.reconstruct(tid, sid, [0.01], S=S, R=60) for S in (1200, 2300))
    assert np.array_equal(rows.category_state, tiles.category_state)
    assert np.array_equal(rows.root_max, tiles.root_max)


@pytest.mark.parametrize("config,K", [(1, 4), (2, 1)])
def test_tile_walk_filter_is_exact(ctx, config, K):
    """k_pupko's log2 filter, which tables past their limit fall back to: the bits
    of the scan of every product."""
    from cafe5_gb300.families import global_bounds
    from cafe5_gb300.inputs import RootPrior, discrete_gamma
    from cafe5_gb300.synth import workload
    w = workload(config, n_families=300, seed=11)
    S, R = global_bounds(w.families)
    tid = ctx.upload_tree(w.tree, w.lambda_of_node)
    sid = ctx.upload_families(tid, w.families.counts)
    ctx.set_prior(RootPrior.uniform(R).vector(R + 8))
    kw = dict(S=S, R=R, lambda_kind=1 if len(w.lambdas) > 1 else 0)
    if K > 1:
        probs, mult = discrete_gamma(0.5, K)
        kw.update(model=1, multipliers=mult, cat_probs=probs)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 1)
    a = ctx.reconstruct(tid, sid, w.lambdas, **kw)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 0)
    b = ctx.reconstruct(tid, sid, w.lambdas, exhaustive=True, **kw)
    for x in ("category_state", "node_count", "node_mean", "root_max", "n_failed"):
        assert np.array_equal(getattr(a, x), getattr(b, x)), x


@pytest.mark.parametrize("newick", ["((A:3.2,B:3.2):4.5,((C:2.5,(D:1.5):1.0):1.25,E:3.75):3.95);",
                                    "(((A:1.5,B:1.5):2.0,C:3.5):1.0);", "((((A:2.0):1.0):0.5,B:3.5):1.0,C:4.5);"],
                         ids=["inside", "root", "chain"])
@pytest.mark.parametrize("eps", [0.0, 0.07])
def test_one_child_nodes(ctx, newick, eps):
    """Nodes with one child, the root among them, against the oracle: global
    bounds and bins 1e-12 relative (two orders of summation), mixed 1e-6."""
    import oracle
    from cafe5_gb300.families import FamilySet, bin_families
    from cafe5_gb300.inputs import ErrorModel, RootPrior
    rng = np.random.default_rng(4)
    n = newick.count(",") + 1
    c = rng.integers(0, 28, (131, n)).astype(np.int32)
    c[:, 0] += 1
    tree, tid, sid = _upload(ctx, newick, c, 40)
    em = ErrorModel.symmetric(eps, int(c.max())) if eps else None
    ctx.set_error_model(em.table() if em else None)
    ta = oracle.TreeArrays.from_tree(tree)
    prior = RootPrior.uniform(40).vector()
    kw = dict(prior=prior, err_rows=em.table() if em else None)
    _, ref, _ = oracle.score(ta, c, [0.01], S=90, R=40, **kw)
    got = ctx.score(tid, sid, [0.01], S=90, R=40, use_error_model=eps > 0).family_lnl
    assert np.all(np.abs(got - ref) <= 1e-12 * np.abs(ref))
    _, Sf, Rf = bin_families(FamilySet([str(i) for i in range(len(c))], c))
    _, binned, _ = oracle.score(ta, c, [0.01], fam_S=Sf, fam_R=Rf, scaled=True, **kw)
    for p, tol in (("fp64_binned", 1e-12), ("mixed_tf32x3", 1e-6)):
        got = ctx.score(tid, sid, [0.01], precision=p, use_error_model=eps > 0).family_lnl
        assert np.all(np.abs(got - binned) <= tol * np.abs(binned)), p
    ctx.set_error_model(None)


@pytest.mark.parametrize("lam,n_sim,R", [(0.3, 40, 30),          # saturated branches: a uniform size first
                                         (0.02, 16385, 2)])      # more than the device sorts
def test_pvalues_drawn_on_the_host(ctx, lam, n_sim, R):
    """The reference's stream where the device does not follow it: against the
    oracle, 1e-10 relative, zeros in the same places."""
    import oracle
    rng = np.random.default_rng(6)
    c = rng.integers(0, 12, (33, 5)).astype(np.int32)
    tree, tid, sid = _upload(ctx, BINARY, c, 60)
    got = ctx.pvalues(tid, sid, [lam], S=60, R=R, n_simulations=n_sim, seed=11)
    pv, cd, rv = oracle.pvalues(oracle.TreeArrays.from_tree(tree), c, [lam], S=60, R=R, n_sim=n_sim, seed=11)
    for x, y in ((got["conditional"], cd), (got["root_likelihood"], rv)):
        assert np.array_equal(x > 0, y > 0)
        assert np.all(np.abs(x - y) <= 1e-10 * y)


@pytest.mark.parametrize("bad", [np.nan, -1.0])
def test_prior_entries_that_are_no_probabilities(ctx, bad):
    """A prior entry that is NaN or negative takes no part in the base model's
    maximum over root sizes (its logarithm is not above any): as if it were 0."""
    rng = np.random.default_rng(7)
    from cafe5_gb300.inputs import RootPrior
    tree, tid, sid = _upload(ctx, BINARY, rng.integers(1, 25, (37, 5)), 60)
    p = RootPrior.uniform(60).vector().copy()
    got = []
    for v in (0.0, bad):
        p[20] = v
        ctx.set_prior(p)
        got.append([ctx.score(tid, sid, [0.01], **kw).family_lnl for kw in
                    (dict(S=90, R=60), dict(precision="fp64_binned"), dict(precision="mixed_tf32x3"))])
    for a, b in zip(*got):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.parametrize("F", [3, 150])           # (units of a few rows, and of eight)
@pytest.mark.parametrize("eps", [-0.05, -0.2])
def test_negative_epsilon(ctx, F, eps):
    """A search over an error model's epsilon may try a negative one: leaf vectors
    are then negative away from the observed count, whole chunks of columns of
    them, and every sum still holds all its terms. At global bounds the bits of the
    tile walk, which forms every product; in bins the oracle's values, 1e-11
    relative (two orders of summation, of terms that partly cancel)."""
    import oracle
    from cafe5_gb300.families import FamilySet, bin_families
    from cafe5_gb300.inputs import RootPrior
    rng = np.random.default_rng(8)
    # C and D pull their parent's vector past state 32, where E's is negative: the
    # node above has its largest values there
    c = rng.integers([22, 22, 35, 35, 18], [31, 31, 38, 38, 24], (F, 5)).astype(np.int32)
    tree, tid, sid = _upload(ctx, BINARY, c, 60)
    table = np.tile([eps, 1 - 2 * eps, eps], (40, 1))
    table[0] = [0.0, 1 - eps, eps]
    ctx.set_error_model(table)
    kw = dict(model=1, multipliers=[0.4, 1.6], cat_probs=[0.5, 0.5])
    score = dict(kw, use_error_model=True, want_categories=True)
    rows = ctx.score(tid, sid, [0.01], S=110, R=60, **score)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 1)
    tiles = ctx.score(tid, sid, [0.01], S=110, R=60, **score)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 0)
    assert np.any(np.isfinite(rows.category_lnl))
    assert np.array_equal(rows.category_lnl, tiles.category_lnl, equal_nan=True)
    assert np.array_equal(rows.family_lnl, tiles.family_lnl, equal_nan=True)
    _, Sf, Rf = bin_families(FamilySet([str(i) for i in range(F)], c))
    _, ref, _ = oracle.score(oracle.TreeArrays.from_tree(tree), c, [0.01], fam_S=Sf, fam_R=Rf, scaled=True,
                             prior=RootPrior.uniform(60).vector(), err_rows=table, **kw)
    got = ctx.score(tid, sid, [0.01], precision="fp64_binned", **score).family_lnl
    ok = np.isfinite(ref)          # (the oracle's NaN: a category whose root values are all negative)
    assert np.all(np.abs(got[ok] - ref[ok]) <= 1e-11 * np.abs(ref[ok]))
    ctx.set_error_model(None)
