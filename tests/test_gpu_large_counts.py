"""Counts far past any state: such a family has probability 0, and the others
of its set keep their results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 0.07])
@pytest.mark.parametrize("huge", [(1 << 14) - 1, 1 << 14, 1 << 30, (1 << 31) - 1])
def test_counts_past_every_state(huge, eps):
    """The tables of a set do not grow with its largest count: 16,383 is the last
    one that is listed by flags, 2^31 - 1 the largest there is. The ordinary
    families' likelihoods are those without the huge one, bit for bit (FP64), or
    within 1e-6 (mixed: its bins' range checks are per family)."""
    from cafe5_gb300.engine import Context
    from cafe5_gb300.inputs import ErrorModel, RootPrior
    from cafe5_gb300.tree import parse_newick
    tree = parse_newick("((A:3.2,B:3.2):4.5,((C:2.5,D:2.5):1.25,E:3.75):3.95);")
    c = np.random.default_rng(1).integers(0, 30, (50, 5), dtype=np.int32)
    c[:, 0] += 1
    h = c.copy()
    h[17, 2] = huge
    keep = np.arange(50) != 17
    ctx = Context(n_streams=1)
    try:
        tid = ctx.upload_tree(tree)
        ctx.set_prior(RootPrior.uniform(40).vector())
        ctx.set_error_model(ErrorModel.symmetric(eps, 40).table() if eps else None)
        small, large = ctx.upload_families(tid, c[keep]), ctx.upload_families(tid, h)
        for p, tol in (("fp64_binned", 0.0), ("mixed_tf32x3", 1e-6)):
            a, b = (ctx.score(tid, s, [0.01], precision=p, use_error_model=eps > 0) for s in (small, large))
            assert np.all(np.isfinite(a.family_lnl))
            assert np.all(np.abs(b.family_lnl[keep] - a.family_lnl) <= tol * np.abs(a.family_lnl)), p
            assert not np.isfinite(b.family_lnl[17]) and b.total == np.inf, p
    finally:
        ctx.close()
