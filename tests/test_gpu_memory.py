"""Calls that run out of device memory (cafe_debug_set, CAFE_DEBUG_ALLOC_LIMIT:
larger buffers are refused on the host) and calls whose tables are split."""
import numpy as np
import pytest

from cafe5_gb300 import _lib

pytestmark = pytest.mark.gpu

OOM = 1


@pytest.fixture
def ctx():
    from cafe5_gb300.engine import Context
    c = Context(n_streams=1)
    yield c
    c.close()


def _limited(ctx, n, call):
    """The call's result with no device buffer over n bytes, or None for out of memory."""
    ctx.debug_set(_lib.DEBUG_ALLOC_LIMIT, n)
    try:
        return call()
    except _lib.CafeError as e:
        assert e.code == OOM, str(e)
        return None
    finally:
        ctx.debug_set(_lib.DEBUG_ALLOC_LIMIT, 0)


@pytest.mark.parametrize("device_sampling", [False, True], ids=["reference stream", "device"])
def test_pvalues_without_room_for_tables(ctx, device_sampling):
    """The simulated families' factor tables (over 16 MB here: 90 root sizes x 500
    families of 12 taxa) are a choice: without them the tile walk runs, and
    without the stream's words the host draws. The same bits either way; where
    even those do not fit, out of memory, and the next call is untouched."""
    from cafe5_gb300.synth import workload
    w = workload(0, n_families=40, seed=4)
    tid = ctx.upload_tree(w.tree)
    sid = ctx.upload_families(tid, w.families.counts)

    def call():
        return ctx.pvalues(tid, sid, [0.0025], S=130, R=90, n_simulations=500, seed=3, device_sampling=device_sampling)

    ref = call()
    done = {}
    for mb in (64, 16, 8, 4, 2, 1, 0.25):
        got = _limited(ctx, int(mb * (1 << 20)), call)
        done[mb] = got is not None
        for r in filter(None, (got, call())):
            for k in ("pvalues", "conditional", "root_likelihood"):
                assert np.array_equal(r[k], ref[k]), (mb, k)
    # (every other buffer takes at most 8 MB: the words, 22 draws of 8 bytes of 45,000 families)
    assert done[16]
    assert device_sampling or done[4]


@pytest.mark.parametrize("F", [40, 6000])
def test_update_that_runs_out_of_memory(ctx, F):
    """A failed cafe_families_update leaves no half-built tables in use: scores are
    refused (invalid), the same update repeated rebuilds everything, and the
    results are those of a set uploaded with these counts. From identical
    families to distinct ones, so that the pattern tables grow."""
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.synth import workload
    w = workload(1, n_families=F, seed=9)
    b = w.families.counts
    a = np.ascontiguousarray(np.tile(b[:1], (F, 1)))
    tid = ctx.upload_tree(w.tree)
    ctx.set_prior(RootPrior.uniform(150).vector())
    modes = [dict(precision="fp64_ref", S=170, R=150), dict(precision="fp64_binned"), dict(precision="mixed_tf32x3")]

    def scores(sid):
        return [ctx.score(tid, sid, [0.002], **m).family_lnl for m in modes]

    fresh = scores(ctx.upload_families(tid, b))
    failed = 0
    for k in range(9, 25):
        sid = ctx.upload_families(tid, a)
        if _limited(ctx, 1 << k, lambda: ctx.update_families(sid, b) or True) is None:
            failed += 1
            for m in modes:
                with pytest.raises(_lib.CafeError) as e:
                    ctx.score(tid, sid, [0.002], **m)
                assert e.value.code == 6
            with pytest.raises(_lib.CafeError) as e:
                ctx.reconstruct(tid, sid, [0.002], S=170, R=150)
            assert e.value.code == 6
            ctx.update_families(sid, b)
        assert all(np.array_equal(x, y) for x, y in zip(scores(sid), fresh))
        ctx.free_families(sid)
    assert failed > 0


def _caterpillar(taxa):
    """A tree with as many levels as internal nodes."""
    from cafe5_gb300.tree import parse_newick
    s = "(T0:1,T1:1)"
    for i in range(2, taxa):
        s = f"({s}:1,T{i}:{i})"
    return parse_newick(s + ";")


def test_tables_of_a_deep_tree(ctx):
    """20,000 families of a tree of 39 levels: a combination's factor table takes
    0.2 GB, and 64 combinations are in flight for one launch. No buffer passes 4
    GB, and every candidate keeps the bits it has alone."""
    from cafe5_gb300.inputs import RootPrior
    c = np.random.default_rng(7).integers(0, 31, (20000, 40), dtype=np.int32)
    tid = ctx.upload_tree(_caterpillar(40))
    sid = ctx.upload_families(tid, c)
    ctx.set_prior(RootPrior.uniform(40).vector())
    kw = dict(model=1, precision="mixed_tf32x3")
    cands = [dict(lambdas=[0.004 * (1 + 0.01 * b)], multipliers=[0.3, 0.7, 1.1, 1.9], cat_probs=[0.25] * 4)
             for b in range(16)]
    got = _limited(ctx, 4 << 30, lambda: ctx.score_batch(tid, sid, cands, **kw))
    assert got is not None
    for b in (0, 9, 15):
        alone = ctx.score(tid, sid, cands[b]["lambdas"], multipliers=cands[b]["multipliers"],
                          cat_probs=cands[b]["cat_probs"], **kw)
        assert np.array_equal(alone.family_lnl, got[b].family_lnl)


def test_fp64_without_room_for_tables(ctx):
    """FP64 tables of 1 GB (0.4 in bins) where no buffer may pass 256 MB: the tile
    walk takes the families, with the same bits (the same chains of sums)."""
    from cafe5_gb300.inputs import RootPrior
    c = np.random.default_rng(8).integers(0, 31, (20000, 40), dtype=np.int32)
    tid = ctx.upload_tree(_caterpillar(40))
    sid = ctx.upload_families(tid, c)
    ctx.set_prior(RootPrior.uniform(40).vector())
    for kw in (dict(precision="fp64_ref", S=170, R=150), dict(precision="fp64_binned"),
               dict(precision="fp64_binned", model=1, multipliers=[0.5, 1.5], cat_probs=[0.4, 0.6])):
        tiles = _limited(ctx, 256 << 20, lambda: ctx.score(tid, sid, [0.004], **kw))
        rows = ctx.score(tid, sid, [0.004], **kw)
        assert tiles is not None
        assert np.array_equal(tiles.family_lnl, rows.family_lnl) and tiles.total == rows.total


@pytest.fixture(params=[1, 100 << 10, 1 << 20], ids=["1 byte", "100 KB", "1 MB"])
def small_tables(ctx, request):
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, request.param)
    yield ctx
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 0)


def _families(F, tree, tail, seed):
    """Random families: counts up to 30, a few up to each of `tail`."""
    rng = np.random.default_rng(seed)
    hi = np.full(F, 30)
    hi[:len(tail)] = tail
    c = rng.integers(0, hi[:, None] + 1, (F, len(tree.leaves))).astype(np.int32)
    c[:, 0] = np.maximum(hi, 1)
    return np.ascontiguousarray(c[rng.permutation(F)])


@pytest.mark.parametrize("F,eps", [(70, 0.0), (70, 0.07), (300, 0.0)])      # (the plan from the host, and the device)
def test_scores_with_tables_split(small_tables, F, eps):
    """The routes of very large sets on a small one: bins in parts (at one byte a
    family each), tables taken over by every next combination, the list of flagged
    terms in passes, FP64 at global bounds by the tile walk. Bins of 64 to 768
    states; the same bits as unsplit."""
    from cafe5_gb300.inputs import ErrorModel, RootPrior
    from cafe5_gb300.synth import workload
    ctx = small_tables
    tree = workload(1, n_families=10, seed=3).tree
    c = _families(F, tree, [60, 60, 100, 150, 200, 300, 380, 600, 610], 5)
    ctx.set_prior(RootPrior.uniform(700).vector())
    ctx.set_error_model(ErrorModel.symmetric(eps, int(c.max())).table() if eps else None)
    tid = ctx.upload_tree(tree)
    split = ctx.upload_families(tid, c)
    limit = {}
    for p, kw in (("fp64_ref", dict(S=620, R=640)), ("fp64_binned", {}), ("mixed_tf32x3", {})):
        for model, extra in ((0, [{}] * 9), (1, [dict(multipliers=[0.3, 0.8, 1.9], cat_probs=[0.2, 0.5, 0.3])] * 9)):
            cands = [dict(e, lambdas=[0.002 * (1 + 0.05 * b)]) for b, e in enumerate(extra)]
            limit[p, model] = (cands, kw, ctx.score_batch(tid, split, cands, model=model, precision=p,
                                                          use_error_model=eps > 0, want_categories=True, **kw))
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 0)
    whole = ctx.upload_families(tid, c)
    for (p, model), (cands, kw, got) in limit.items():
        ref = ctx.score_batch(tid, whole, cands, model=model, precision=p, use_error_model=eps > 0, want_categories=True,
                              **kw)
        for a, b in zip(got, ref):
            assert a.status == b.status and a.n_fallback == b.n_fallback, p
            assert np.array_equal(a.family_lnl, b.family_lnl, equal_nan=True), p
            assert np.array_equal(a.category_lnl, b.category_lnl, equal_nan=True), p
            assert a.total == b.total or (np.isnan(a.total) and np.isnan(b.total)), p
    ctx.set_error_model(None)


def test_reconstruction_with_tables_split(small_tables):
    """Categories in passes, and the tile walk where one category's tables pass the
    limit: the same states, counts and root values."""
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.synth import workload
    ctx = small_tables
    tree = workload(1, n_families=10, seed=3).tree
    c = _families(150, tree, [], 6)
    ctx.set_prior(RootPrior.uniform(60).vector())
    tid = ctx.upload_tree(tree)
    sid = ctx.upload_families(tid, c)
    kw = dict(S=80, R=60, model=1, multipliers=[0.2, 0.6, 1.1, 2.1], cat_probs=[0.25] * 4)
    got = ctx.reconstruct(tid, sid, [0.002], **kw)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 12 << 20)      # (between one category's tables, 5 MB, and all four's)
    passes = ctx.reconstruct(tid, sid, [0.002], **kw)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, 0)
    for ref in (ctx.reconstruct(tid, sid, [0.002], **kw), ctx.reconstruct(tid, sid, [0.002], exhaustive=True, **kw)):
        for a in (got, passes):
            assert np.array_equal(a.category_state, ref.category_state) and np.array_equal(a.node_count, ref.node_count)
            assert np.array_equal(a.root_max, ref.root_max) and np.array_equal(a.node_mean, ref.node_mean)
            assert a.n_failed == ref.n_failed


@pytest.mark.parametrize("kb", [1, 8 << 10, 32 << 10])      # (the tile walk; many passes; a few)
def test_pvalues_with_tables_split(ctx, kb):
    """Simulated families in several passes of state bounds, or by the tile walk
    where one bound's tables pass the limit; observed ones by the tile walk."""
    from cafe5_gb300.synth import workload
    w = workload(0, n_families=300, seed=4)
    tid = ctx.upload_tree(w.tree)
    sid = ctx.upload_families(tid, w.families.counts)
    kw = dict(S=200, R=90, n_simulations=400, seed=3)      # (state bounds 51 to about 150)
    ref = ctx.pvalues(tid, sid, [0.0025], **kw)
    ctx.debug_set(_lib.DEBUG_TABLE_BYTES, kb << 10)
    got = ctx.pvalues(tid, sid, [0.0025], **kw)
    for k in ("pvalues", "conditional", "root_likelihood"):
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("kw", [dict(precision="mixed_tf32x3"), dict(precision="fp64_binned"),
                                dict(precision="fp64_ref", S=170, R=150)], ids=lambda k: k["precision"])
def test_serving_counts_the_tables(kw):
    """The request loop's budget covers the factor tables: 10,000 families of 24
    taxa take 3 MB of results and over 10 MB of tables a category, so with a budget
    of 40 MB two requests of four categories (on two sets: they share no launch) never run
    side by side, which they do without it."""
    from cafe5_gb300.engine import Context
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.synth import workload
    w = workload(1, n_families=10000, seed=36)
    ctx = Context()
    try:
        ctx.set_prior(RootPrior.uniform(150).vector())
        tid = ctx.upload_tree(w.tree)
        sets = [ctx.upload_families(tid, w.families.counts) for _ in range(2)]
        kw = dict(kw, model=1, multipliers=w.multipliers, cat_probs=w.cat_probs)
        ref = [ctx.score(tid, s, [0.002], **kw).total for s in sets]

        def overlap():
            before = ctx.serving_stats()["overlap_ms"]
            handles = [ctx.submit(tid, sets[i % 2], [0.002], **kw) for i in range(12)]
            got = np.array([ctx.poll(h).total for h in handles])
            assert np.all(np.abs(got - ref * 6) <= 1e-6 * got)
            return ctx.serving_stats()["overlap_ms"] - before

        assert any(overlap() > 0 for _ in range(5))
        ctx.debug_set(_lib.DEBUG_SERVE_BUDGET, 40 << 20)
        assert overlap() == 0
    finally:
        ctx.close()
