"""What many calls on one context leave behind."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _resident_bytes():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGESIZE")


def test_fp64_scores_keep_host_memory():
    """The host keeps no record of a call that is not part of a CUDA graph. An
    FP64 score issues about ten stream operations with the arguments of two
    kernels, over 500 bytes: 30,000 scores would leave 15 MB behind. Allowed: 4
    MB, for the allocator and the driver."""
    from cafe5_gb300.engine import Context
    from cafe5_gb300.inputs import RootPrior
    from cafe5_gb300.tree import parse_newick
    ctx = Context(n_streams=1)
    try:
        tid = ctx.upload_tree(parse_newick("((A:3.2,B:3.2):4.5,C:7.7);"))
        sid = ctx.upload_families(tid, np.array([[1, 2, 1], [3, 1, 2]], np.int32))
        ctx.set_prior(RootPrior.uniform(20).vector())
        kw = dict(S=20, R=20)
        first = ctx.score(tid, sid, [0.01], **kw)
        for _ in range(2000):
            ctx.score(tid, sid, [0.01], **kw)
        before = _resident_bytes()
        for _ in range(30000):
            last = ctx.score(tid, sid, [0.01], **kw)
        assert _resident_bytes() - before <= 4 << 20
        assert np.array_equal(first.family_lnl, last.family_lnl)
    finally:
        ctx.close()
