"""GPU parity of the two-pairs-per-thread banded kernel with the one-pair kernel (every field and
segment) and the oracle (scores): bands of 2 to 41 diagonals in every position -- through the origin,
right and left of it, wider than the matrix, leaving it at the bottom or on the right -- batches
of pairs that share a thread, odd ones out and padding, every AlignConfig, linear and affine gaps,
tables, and pairs at the edge of the value range."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _batch(rng, sizes, alphabet=4):
    H, V = [], []
    for m, n, count in sizes:
        for _ in range(count):
            h = rng.integers(0, alphabet, m).astype(np.uint8)
            v = rng.integers(0, alphabet, n).astype(np.uint8)
            at = int(rng.integers(0, max(1, m - n // 2)))
            k = min(n, m - at)
            v[:k] = h[at:at + k]
            v[rng.random(n) < 0.1] = 1
            H.append(h)
            V.append(v)
    order = rng.permutation(len(H))
    return [H[i] for i in order], [V[i] for i in order]


def _compare(H, V, score, cfg, band, alphabet, traceback=True):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    new = sg.align_codes(H, V, score, config=cfg, band=band, traceback=traceback, cigar=traceback, alphabet_size=alphabet)
    old = sg.align_codes(H, V, score, config=cfg, band=band, traceback=traceback, cigar=traceback, alphabet_size=alphabet,
                         flags=N.GBA_FLAG_GENERAL_KERNEL)
    for f in ("score", "end_h", "end_v", "status") + (("begin_h", "begin_v", "segment_offsets", "cigar_offsets")
                                                      if traceback else ()):
        assert np.array_equal(getattr(new, f), getattr(old, f)), f
    if traceback:
        assert np.array_equal(new.segments[:new.segment_offsets[-1]], old.segments[:old.segment_offsets[-1]])
        assert np.array_equal(new.cigar[:new.cigar_offsets[-1]], old.cigar[:old.cigar_offsets[-1]])
    return new


@pytest.mark.parametrize("scheme", [(2, -4, -6, -1), (2, -3, -5, -5), (3, -2, -1, -4), (5, -1, 0, 0), (1, -1, -2, 0)])
@pytest.mark.parametrize("fe", range(16))
def test_bands(engine, scheme, fe):
    import seqan_gb300 as sg
    mt, mm, go, ge = scheme
    rng = np.random.default_rng(31 * fe + mt)
    score = sg.Score(mt, mm, ge, go, dtype=np.int16)
    cfg = sg.AlignConfig(bool(fe & 1), bool(fe & 2), bool(fe & 4), bool(fe & 8))
    for w in (2, 3, 8, 9, 32, 33, 40, 41):
        for lo in (-w + 1, -w // 2, 0, 4, -w - 3):
            sizes = [(60, 50, 5), (50, 60, 2), (70, 40, 1), (45, 45, 3), (12, 30, 2), (30, 9, 2), (1, 5, 2), (6, 1, 2),
                     (41, 40, 4)]
            H, V = _batch(rng, sizes)
            out = _compare(H, V, score, cfg, (lo, lo + w - 1), 4)
            ref = O.oracle_batch(O.Problem(free_ends=fe, band=(lo, lo + w - 1), match=mt, mismatch=mm, gap_open=go,
                                           gap_extend=ge, score_bits=16), H, V)
            assert out.score.tolist() == ref.score.tolist(), (w, lo)


@pytest.mark.parametrize("count", [1, 2, 63, 64, 65, 130])
def test_groups(engine, count):
    """Group sizes of the 64-slot layout, with the odd pair on the one-pair kernel."""
    import seqan_gb300 as sg
    rng = np.random.default_rng(count)
    H, V = _batch(rng, [(120, 100, count)])
    for tb in (False, True):
        _compare(H, V, sg.Score(2, -4, -1, -6, dtype=np.int16), sg.AlignConfig(True, False, False, True), (-6, 26), 4, tb)


@pytest.mark.parametrize("scale", [1, 12, 93, 94])
def test_tables(engine, scale):
    import seqan_gb300 as sg
    rng = np.random.default_rng(scale)
    score = sg.Blosum62(-1, -11)
    score.matrix = np.ascontiguousarray(score.matrix * scale)
    H, V = _batch(rng, [(90, 80, 40), (80, 90, 3)], 26)
    for fe in (0, 9):
        cfg = sg.AlignConfig(bool(fe & 1), False, False, bool(fe & 8))
        _compare(H, V, score, cfg, (-12, 15), 27)


@pytest.mark.parametrize("bits", [16, 32])
@pytest.mark.parametrize("scheme,length", [((100, -100, -200, -50), 138), ((100, -100, -200, -50), 142),
                                           ((2, -4, -6, -1), 2600), ((2, -4, -6, -1), 2680)])
def test_range_edge(engine, bits, scheme, length):
    """The last pairs inside the value range and the first ones beyond it."""
    import seqan_gb300 as sg
    mt, mm, go, ge = scheme
    rng = np.random.default_rng(length)
    H, V = _batch(rng, [(length, length, 4), (length + 8, length, 4)])
    H[0][:], V[0][:] = 2, 2          # the best score
    H[1][:], V[1][:] = 2, 3          # the worst
    for fe in (0, 15):
        cfg = sg.AlignConfig(*(bool(fe),) * 4)
        _compare(H, V, sg.Score(mt, mm, ge, go, dtype=np.int16 if bits == 16 else np.int32), cfg, (-10, 14), 4)
