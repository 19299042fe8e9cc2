"""GPU parity of GappedXDrop seed extension with the oracle where a live range fills its ring: drop-offs
at the last of each ring size and the first of the next (12 / 13, 28 / 29, 60 / 61 gaps), tiny and
empty sides, high-scoring pairs whose ranges grow past 16, 32 and 64 columns, and drop-offs of zero."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap,mismatch,match", [(-1, -1, 1), (-3, -2, 2), (-1, -1, 3)])
@pytest.mark.parametrize("gaps,ring", [(0, 16), (1, 16), (5, 16), (12, 16), (13, 32), (28, 32), (29, 64), (60, 64),
                                       (61, 0)])
def test_rings(engine, gap, mismatch, match, gaps, ring):
    import seqan_gb300 as sg
    from seqan_gb300 import seeds as S
    from seqan_gb300 import workloads as W
    rng = np.random.default_rng(10 * gaps + match)
    H, V, seeds = [], [], []
    for k in range(700):
        h = rng.integers(0, 4 if k % 3 else 2, int(rng.choice([1, 2, 3, 15, 17, 40, 150, 260]))).astype(np.uint8)
        v = W.mutate(rng, h, float(rng.uniform(0, 0.3)), float(rng.uniform(0, 0.1)))
        if k % 4 == 0 or len(v) == 0:
            v = rng.integers(0, 4, int(rng.choice([1, 2, 30, 200]))).astype(np.uint8)
        at = int(rng.integers(0, min(len(h), len(v)) + 1))
        H.append(h)
        V.append(v)
        seeds.append((at, at, 0))
    sp = O.SeedProblem(O.GAPPED_XDROP, O.EXTEND_BOTH, match, mismatch, gap, gaps * -gap)
    arr = O.seeds_array(seeds)
    got, xs = S.extend_seeds(arr, H, V, sp.direction, sg.Score(match, mismatch, gap), sp.xdrop, sp.method,
                             alphabet="dna5", return_scores=True)
    assert sg.default_context().stats().seed_ring == ring
    ref, rx = O.oracle_extend_seeds(sp, H, V, arr)
    assert np.array_equal(got, ref)
    assert np.array_equal(xs, rx)
