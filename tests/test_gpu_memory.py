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
