"""Pattern plans built on the host (small sets) and on the device: the same
rows, so the same bits of every result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BINARY = "((A:3.2,B:3.2):4.5,((C:2.5,D:2.5):1.25,E:3.75):3.95);"
POLY = "((A:3.2,B:3.2,C:3.2):4.5,(D:2.5,(E:1.5):1.0,F:2.5):5.2,G:7.7);"


@pytest.mark.parametrize("newick,nodes", [(BINARY, 4), (POLY, 4), ("(A:1.0,B:2.0);", 1)],
                         ids=["binary", "polytomy", "root only"])
@pytest.mark.parametrize("hi", [9, 90])           # one bin, and several
def test_host_and_device_plans(newick, nodes, hi):
    """Families x internal nodes on both sides of the 6,000 up to which the host
    builds the plan: a set just above holds a set just below as its first
    families."""
    from cafe5_gb300.engine import Context
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick(newick)
    rng = np.random.default_rng([hi, nodes])
    F = 6000 // nodes
    c = rng.integers(0, hi + 1, (F + 1, len(tree.leaves)), dtype=np.int32)
    c = np.minimum(c, rng.integers(1, hi + 1, (F + 1, 1))).astype(np.int32)      # (families of every size)
    c[:, 0] = np.maximum(c[:, 0], 1)
    c[0] = hi
    ctx = Context(n_streams=1)
    try:
        tid = ctx.upload_tree(tree)
        ctx.set_prior(RootPrior.uniform(60).vector())
        host, device = ctx.upload_families(tid, c[:F]), ctx.upload_families(tid, c)
        for kw in (dict(precision="fp64_ref", S=110, R=60), dict(precision="fp64_binned"),
                   dict(precision="mixed_tf32x3")):
            a, b = (ctx.score(tid, s, [0.01], **kw) for s in (host, device))
            assert np.all(np.isfinite(a.family_lnl))
            assert np.array_equal(a.family_lnl, b.family_lnl[:F]), kw
        a, b = (ctx.reconstruct(tid, s, [0.01], S=110, R=60) for s in (host, device))
        assert np.array_equal(a.node_count, b.node_count[:F]) and np.array_equal(a.root_max, b.root_max[:, :F])
    finally:
        ctx.close()


def test_upload_of_a_small_set_is_quick():
    """A plan on the device costs a small set several launches and round trips
    (an upload of 100 families of 8 taxa took 240 us, 57 without plans, 42 with
    one from the host). Median of 50; the limit is three times the latter, for a
    slower host."""
    import time
    from cafe5_gb300 import synth
    from cafe5_gb300.engine import Context
    tree = synth.yule_tree(8, 60.0, 1)
    c = np.random.default_rng(2).integers(1, 12, (100, 8), dtype=np.int32)
    ctx = Context(n_streams=1)
    try:
        tid = ctx.upload_tree(tree)
        took = []
        for _ in range(50):
            t = time.perf_counter()
            sid = ctx.upload_families(tid, c)
            took.append(time.perf_counter() - t)
            ctx.free_families(sid)
        assert sorted(took)[25] <= 126e-6
    finally:
        ctx.close()
