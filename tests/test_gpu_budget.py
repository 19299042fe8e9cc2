"""GPU: HBM budgets and the packed 16-bit warp kernel.  A pair whose scratch fits the budget on the
32-bit warp kernel alone is taken, and gives the same result there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _align(h, v, mode, traceback, budget, flags=0):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    ctx = N.Context(0, budget)
    out = sg.align_codes([h], [v], sg.Score(2, -4, -1, -6), mode=mode, traceback=traceback, alphabet_size=4, flags=flags,
                         ctx=ctx)
    return out, ctx.stats().dp_kernels


def _smallest(accepted, high):
    """The smallest budget that is accepted (0: none is set)."""
    low = 0
    while high - low > 1:
        mid = (low + high) // 2
        if accepted(mid):
            high = mid
        else:
            low = mid
    return high


@pytest.mark.parametrize("mode,traceback,m,n", [(0, True, 3000, 16), (1, True, 3000, 16), (1, True, 500, 33),
                                                (0, False, 9000, 200), (0, True, 2000, 700)])
def test_smallest_budget(engine, mode, traceback, m, n):
    from seqan_gb300 import _native as N
    rng = np.random.default_rng(m + n)
    h, v = rng.integers(0, 4, m).astype(np.uint8), rng.integers(0, 4, n).astype(np.uint8)

    def accepted(budget, flags=0):
        try:
            _align(h, v, mode, traceback, budget, flags)
        except RuntimeError as e:
            assert "budget" in str(e)
            return False
        return True

    narrow = _smallest(lambda b: accepted(b, N.GBA_FLAG_NO_WARP16), 64 << 20)
    both = _smallest(accepted, 64 << 20)
    assert both <= narrow
    ref, kernels = _align(h, v, mode, traceback, 0)
    assert kernels & N.GBA_KERNEL_WARP16
    for budget in (both, narrow):
        out, _ = _align(h, v, mode, traceback, budget)
        assert out.score.tolist() == ref.score.tolist()
        if traceback:
            assert out.pair_segments(0) == ref.pair_segments(0)
