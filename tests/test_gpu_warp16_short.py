"""GPU: large batches of pairs of few columns run on the 32-bit warp kernel, smaller ones and ones with a
longer pair on the packed 16-bit one, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,longest,packed", [(16384, 16, False), (16384, 17, True), (16383, 16, True)])
@pytest.mark.parametrize("mode", [0, 1])
def test_short_pairs(engine, count, longest, packed, mode):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    rng = np.random.default_rng(count + longest)
    H = [rng.integers(0, 4, int(m)).astype(np.uint8) for m in rng.integers(1, 17, count)]
    H[count // 2] = rng.integers(0, 4, longest).astype(np.uint8)
    V = [rng.integers(0, 4, int(n)).astype(np.uint8) for n in rng.integers(1, 41, count)]
    score = sg.Score(2, -4, -1, -6)
    out = sg.align_codes(H, V, score, mode=mode, traceback=True, alphabet_size=4)
    kernels = sg.default_context().stats().dp_kernels
    assert bool(kernels & N.GBA_KERNEL_WARP16) == packed and bool(kernels & N.GBA_KERNEL_WARP) != packed
    ref = sg.align_codes(H, V, score, mode=mode, traceback=True, alphabet_size=4, flags=N.GBA_FLAG_NO_WARP16)
    for f in ("score", "end_h", "end_v", "begin_h", "begin_v", "segment_offsets"):
        assert np.array_equal(getattr(out, f), getattr(ref, f)), f
    assert np.array_equal(out.segments[:out.segment_offsets[-1]], ref.segments[:ref.segment_offsets[-1]])
