"""GPU: extendAlignment under an HBM budget: a batch whose two-sides-per-thread form needs more than the
budget runs on the groups' form, with the same results."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget,paired", [(1 << 20, False), (64 << 20, False), (8 << 30, True), (0, True)])
def test_budget(engine, budget, paired):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    from seqan_gb300 import align_extend as X
    rng = np.random.default_rng(5)
    n = 20_000
    H = rng.integers(0, 4, (n, 150)).astype(np.uint8)
    V = H.copy()
    V[rng.random(V.shape) < 0.1] = 1
    pos = [(70, 70, 80, 80)] * n
    score = sg.Score(2, -4, -1, -6)
    ref = X.extend_alignments(list(H), list(V), pos, O.EXTEND_BOTH, score, 15)
    assert N.default_context().stats().tile_rows == 16      # two sides per thread
    ctx = N.Context(0, budget)
    got = X.extend_alignments(list(H), list(V), pos, O.EXTEND_BOTH, score, 15, context=ctx)
    assert (ctx.stats().tile_rows == 16) == paired
    assert got == ref
