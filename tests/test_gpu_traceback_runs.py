"""GPU parity of the warp traceback (k_traceback_warp) where its reads of 32 cells begin and end:
diagonal and gap runs of one less, exactly and one more than one and two reads, at the start, inside
and at the end of the alignment, in both warp layouts (32-bit and packed 16-bit), against the
oracle's TraceSegment_ lists."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

RUNS = [1, 31, 32, 33, 34, 63, 64, 65, 66]


def _pairs(seed):
    """Runs of the lengths in RUNS: a diagonal of each, a gap of each, in either sequence."""
    rng = np.random.default_rng(seed)
    H, V = [], []
    for gap in RUNS:
        for lead in (RUNS[(gap * 5) % len(RUNS)], 40):
            h = rng.integers(0, 4, lead + gap + 70).astype(np.uint8)
            v = np.concatenate([h[:lead], h[lead + gap:]])
            H += [h, v]
            V += [v, h]
    return H, V


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("fe", [0, 15])
@pytest.mark.parametrize("scheme", [(2, -4, -6, -1), (5, -4, -1, -1)])
def test_traceback_runs(engine, packed, fe, scheme):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    match, mismatch, go, ge = scheme
    H, V = _pairs(11 + fe)
    cfg = sg.AlignConfig(bool(fe & 1), bool(fe & 2), bool(fe & 4), bool(fe & 8))
    ref = O.oracle_batch(O.Problem(free_ends=fe, match=match, mismatch=mismatch, gap_open=go, gap_extend=ge,
                                   score_bits=16), H, V, traceback=True)
    out = sg.align_codes(H, V, sg.Score(match, mismatch, ge, go, dtype=np.int16), config=cfg, traceback=True,
                         alphabet_size=4, flags=N.GBA_FLAG_WARP16 if packed else N.GBA_FLAG_NO_WARP16)
    assert bool(sg.default_context().stats().dp_kernels & N.GBA_KERNEL_WARP16) == packed
    assert out.score.tolist() == ref.score.tolist()
    for k in range(len(H)):
        assert out.pair_segments(k) == ref.segments[k], k
