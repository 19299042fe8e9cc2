"""GPU parity of the Waterman-Eggert enumerator with the oracle on both sides of its two sizes: batches
whose largest pair has 128 cells (a thread per pair) and 129 (a warp per pair), 1,024 cells (pairs as
they come) and 1,025 (the largest first), the largest pair first, last and inside."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(15, 7), (7, 15), (42, 2), (2, 42), (31, 31), (40, 24), (24, 40)])
@pytest.mark.parametrize("at", [0, 20, 39])
def test_sizes(engine, m, n, at):
    import seqan_gb300 as sg
    from seqan_gb300 import local_enum as LE
    rng = np.random.default_rng(100 * m + at)
    H = [rng.integers(0, 2, int(rng.integers(0, m + 1))).astype(np.uint8) for _ in range(40)]
    V = [rng.integers(0, 2, int(rng.integers(0, n + 1))).astype(np.uint8) for _ in range(40)]
    H[at], V[at] = rng.integers(0, 2, m).astype(np.uint8), rng.integers(0, 2, n).astype(np.uint8)
    got = LE.local_enumerate(H, V, sg.Score(2, -1, -2, -2), 3, 6, alphabet="dna5")
    for k in range(40):
        ref = O.oracle_local_enumerate(H[k], V[k], 2, -1, -2, 3, max_count=6)
        undefined = bool(ref) and ref[-1] is None
        ref = ref[:-1] if undefined else ref
        assert got[k].undefined_next == undefined, k
        assert [(a.score, a.segments) for a in got[k].alignments] == [(a.score, a.segments) for a in ref], k
