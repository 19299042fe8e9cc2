"""GPU parity of the packed 16-bit warp kernel's choices, against the oracle: row counts at the edges
of every rows-per-strip instance and of one, two and three bands, columns around the 64-step front,
in-order and pipelined bands; pairs at the edge of the 16-bit range (the last ones inside and the
first ones on the 32-bit kernel), 32-bit score types, tables of byte, wide and too wide entries, and
codes outside the table's alphabet."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROWS = [1, 63, 64, 127, 128, 129, 192, 193, 256, 257, 320, 321, 384, 385, 512, 513, 768, 1025]


def _run(H, V, score, mode, fe, pb, alphabet, traceback, flags=0):
    import seqan_gb300 as sg
    cfg = sg.AlignConfig(bool(fe & 1), bool(fe & 2), bool(fe & 4), bool(fe & 8)) if mode == 0 else None
    ref = O.oracle_batch(pb, H, V, traceback=traceback)
    out = sg.align_codes(H, V, score, mode=mode, config=cfg, traceback=traceback, alphabet_size=alphabet, flags=flags)
    assert out.score.tolist() == ref.score.tolist()
    assert out.end_h.tolist() == ref.end_h.tolist() and out.end_v.tolist() == ref.end_v.tolist()
    if traceback:
        for k in range(len(H)):
            assert out.pair_segments(k) == ref.segments[k], k
    return sg.default_context().stats().dp_kernels


def _pairs(seed, rows, alphabet=4):
    rng = np.random.default_rng(seed)
    H, V = [], []
    for n in rows:
        for m in (1, 63, 64, 65, 130, n):
            v = rng.integers(0, alphabet, n).astype(np.uint8)
            h = rng.integers(0, alphabet, m).astype(np.uint8)
            k = min(m, n) * 3 // 4
            h[m - k:] = v[:k]
            H.append(h)
            V.append(v)
    return H, V


@pytest.mark.parametrize("traceback", [False, True])
@pytest.mark.parametrize("mode,fe", [(0, 0), (0, 5), (0, 15), (1, 0)])
@pytest.mark.parametrize("scheme", [(2, -4, -6, -1), (2, -3, -5, -5)])
def test_rows(engine, traceback, mode, fe, scheme):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    mt, mm, go, ge = scheme
    pb = O.Problem("local" if mode else "global", fe, None, mt, mm, go, ge, None, 16)
    score = sg.Score(mt, mm, ge, go, dtype=np.int16)
    H, V = _pairs(3 + fe, ROWS)
    assert _run(H, V, score, mode, fe, pb, 4, traceback) & N.GBA_KERNEL_WARP16
    # few pairs: the longest ones run their bands on several warps
    for k in (len(H) - 1, len(H) - 13):
        _run([H[k]], [V[k]], score, mode, fe, pb, 4, traceback)
    # the plain form keeps a pair's bands on one warp
    _run(H * 8, V * 8, score, mode, fe, pb, 4, traceback, N.GBA_FLAG_PLAIN_BUCKETS)


@pytest.mark.parametrize("bits", [16, 32])
@pytest.mark.parametrize("length", [3098, 3099, 3100, 3101, 3102, 3200])
def test_range_edge(engine, bits, length):
    """Global scores with extension -5: the 16-bit range ends at about 6,200 residues a pair."""
    import seqan_gb300 as sg
    rng = np.random.default_rng(length)
    H = [rng.integers(0, 4, length).astype(np.uint8) for _ in range(3)]
    V = [rng.integers(0, 4, length).astype(np.uint8), np.zeros(length, np.uint8), H[2].copy()]
    H[1][:] = 1
    H[1][5:900] = 0   # all gaps but one stretch
    pb = O.Problem("global", 0, None, 2, -4, -6, -5, None, 32)
    dt = np.int16 if bits == 16 else np.int32
    _run(H, V, sg.Score(2, -4, -5, -6, dtype=dt), 0, 0, pb, 4, True)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("scale", [1, 11, 12, 93, 94])
def test_tables(engine, mode, scale):
    """Blosum62 scaled: entries fit a byte (up to 11 * 11), a table of 1,024 (up to 93), neither."""
    import seqan_gb300 as sg
    score = sg.Blosum62(-1, -11)
    score.matrix = np.ascontiguousarray(score.matrix * scale)
    H, V = _pairs(scale, [1, 100, 128, 129, 300, 390], 24)
    pb = O.Problem("local" if mode else "global", 0, None, 0, 0, -11, -1, score.matrix, 32, "aa")
    _run(H, V, score, mode, 0, pb, 27, True)


def test_codes_outside_alphabet(engine):
    """Codes at or above the table's alphabet score 0, on every kernel."""
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    score = sg.Blosum62(-1, -11)
    score.matrix = np.ascontiguousarray(score.matrix[:20, :20])
    H, V = _pairs(9, [64, 200, 400], 26)
    for mode in (0, 1):
        a = sg.align_codes(H, V, score, mode=mode, traceback=True)
        assert sg.default_context().stats().dp_kernels & N.GBA_KERNEL_WARP16
        b = sg.align_codes(H, V, score, mode=mode, traceback=True, flags=N.GBA_FLAG_GENERAL_KERNEL)
        assert a.score.tolist() == b.score.tolist()
        assert [a.pair_segments(k) for k in range(len(H))] == [b.pair_segments(k) for k in range(len(H))]
