"""GPU: what the server counts for a request covers what the packed 16-bit warp kernel allocates for it,
and a request that fits the budget on the 32-bit warp kernel alone is taken and runs there."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _serve(h, v, budget, **options):
    import seqan_gb300 as sg
    from seqan_gb300.serving import Server
    with Server(sg.Score(2, -4, -1, -6), streams=1, max_batch_pairs=16, hbm_budget_bytes=budget, alphabet_size=4,
                **options) as srv:
        assert srv.submit(7, h, v) == 0
        done = []
        t0 = time.time()
        while not done:
            done = srv.poll()
            assert time.time() - t0 < 60
        return done[0], srv.stats().hbm_in_flight_peak


def _pair(m, n):
    rng = np.random.default_rng(m + n)
    return rng.integers(0, 4, m).astype(np.uint8), rng.integers(0, 4, n).astype(np.uint8)


@pytest.mark.parametrize("n", [129, 200, 256, 257, 700])
def test_row_buffers_are_counted(engine, n):
    """More than one band of 128 rows: two rows of 8-byte entries, whatever the trace."""
    m = 9000
    _, counted = _serve(*_pair(m, n), 1 << 30, traceback=False)
    assert counted >= m + n + 16 * (m + 1)


@pytest.mark.parametrize("mode", [0, 1])
def test_request_that_fits_the_32_bit_kernel_alone(engine, mode):
    import seqan_gb300 as sg
    m, n = 3000, 16
    h, v = _pair(m, n)
    # row 0's trace, m + 32 steps of 128 bytes, two arrays of segment slots, the codes and a few words
    budget = (m + 16) + (m + 32) * 128 + (m + n + 4) * 32 + m + n + 512
    got, peak = _serve(h, v, budget, mode=mode)
    assert peak <= budget
    ref = sg.align_codes([h], [v], sg.Score(2, -4, -1, -6), mode=mode, traceback=True, alphabet_size=4)
    assert got.status == 0 and got.score == ref.score[0] and got.segments == ref.pair_segments(0)
