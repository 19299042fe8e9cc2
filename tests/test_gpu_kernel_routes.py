"""GPU: which kernel a call takes on both sides of each rule that chooses one (gba_stats.dp_kernels), and
that its results are the other kernel's: banded pairs two per thread, pipelined bands of the packed
16-bit warp kernel and the ends of its value range, the enumerator's warp per pair and the extension's
two sides per thread."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernels():
    import seqan_gb300 as sg
    return sg.default_context().stats().dp_kernels


def _same(a, b):
    for f in ("score", "end_h", "end_v", "begin_h", "begin_v", "segment_offsets"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert np.array_equal(a.segments[:a.segment_offsets[-1]], b.segments[:b.segment_offsets[-1]])


def _pairs(rng, m, n, count):
    H = [rng.integers(0, 4, m).astype(np.uint8) for _ in range(count)]
    V = [rng.integers(0, 4, n).astype(np.uint8) for _ in range(count)]
    for h, v in zip(H, V):
        k = min(m, n) * 2 // 3
        v[:k] = h[:k]
    return H, V


# Scheme (match, mismatch, open, extend) and length: the last and first lengths around the best score
# (127 * 110 = 13,970 of 14,000) and around the worst one (3 * 200 + 50 * (2 * 76 + 2) + 100 * 76 = 15,900;
# 3 * 6 + 2 * 2,663 + 2 + 4 * 2,663 = 15,998).
@pytest.mark.parametrize("bits", [16, 32])
@pytest.mark.parametrize("fe", [0, 9, 15])
@pytest.mark.parametrize("scheme,length,duo", [((127, -1, -2, -1), 110, True), ((127, -1, -2, -1), 111, False),
                                               ((100, -100, -200, -50), 76, True), ((100, -100, -200, -50), 77, False),
                                               ((2, -4, -6, -1), 2663, True), ((2, -4, -6, -1), 2664, False)])
def test_banded_value_range(engine, bits, fe, scheme, length, duo):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    mt, mm, go, ge = scheme
    rng = np.random.default_rng(length)
    H, V = _pairs(rng, length, length, 6)
    H[0][:], V[0][:] = 2, 2          # the best score
    H[1][:], V[1][:] = 2, 3          # the worst
    score = sg.Score(mt, mm, ge, go, dtype=np.int16 if bits == 16 else np.int32)
    cfg = sg.AlignConfig(bool(fe & 1), bool(fe & 2), bool(fe & 4), bool(fe & 8))
    for band in ((-5, 5), (-10, 14), (-1, 2)):
        out = sg.align_codes(H, V, score, config=cfg, band=band, traceback=True, alphabet_size=4)
        assert bool(_kernels() & N.GBA_KERNEL_BANDED2) == duo
        _same(out, sg.align_codes(H, V, score, config=cfg, band=band, traceback=True, alphabet_size=4,
                                  flags=N.GBA_FLAG_GENERAL_KERNEL))
        assert not _kernels() & N.GBA_KERNEL_BANDED2


@pytest.mark.parametrize("sizes,band,alphabet,duo", [
    ([(60, 50)] * 2, (0, 1), 4, True), ([(60, 50)], (0, 1), 4, False), ([(60, 50), (60, 51)], (0, 1), 4, False),
    ([(60, 50)] * 2, (0, 39), 4, True), ([(60, 50)] * 2, (0, 40), 4, False), ([(60, 50)] * 2, (3, 3), 4, False),
    ([(60, 50)] * 2, (0, 9), 8, True), ([(60, 50)] * 2, (0, 9), 9, False)])
def test_banded_shapes(engine, sizes, band, alphabet, duo):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    rng = np.random.default_rng(3)
    H = [rng.integers(0, 4, m).astype(np.uint8) for m, _ in sizes]
    V = [rng.integers(0, 4, n).astype(np.uint8) for _, n in sizes]
    cfg = sg.AlignConfig(True, True, True, True)
    out = sg.align_codes(H, V, sg.Score(2, -4, -1, -6), config=cfg, band=band, traceback=True, alphabet_size=alphabet)
    assert bool(_kernels() & N.GBA_KERNEL_BANDED2) == duo and _kernels() & N.GBA_KERNEL_BANDED
    _same(out, sg.align_codes(H, V, sg.Score(2, -4, -1, -6), config=cfg, band=band, traceback=True,
                              alphabet_size=alphabet, flags=N.GBA_FLAG_GENERAL_KERNEL))


@pytest.mark.parametrize("traceback", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("length,count,pipelined", [(60, 1, False), (900, 1, True), (900, 4000, False), (3000, 3, True)])
def test_pipelined_bands(engine, mode, length, count, pipelined, traceback):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    H, V = _pairs(np.random.default_rng(length), length, length - 7, min(count, 10))
    H, V = H * (count // len(H)), V * (count // len(V))
    score = sg.Score(2, -4, -1, -6)
    out = sg.align_codes(H, V, score, mode=mode, traceback=traceback, alphabet_size=4)
    assert _kernels() & N.GBA_KERNEL_WARP16 and bool(_kernels() & N.GBA_KERNEL_PIPELINED) == pipelined
    ref = sg.align_codes(H, V, score, mode=mode, traceback=traceback, alphabet_size=4, flags=N.GBA_FLAG_NO_WARP16)
    assert not _kernels() & (N.GBA_KERNEL_WARP16 | N.GBA_KERNEL_PIPELINED)
    if traceback:
        _same(out, ref)
    assert out.score.tolist() == ref.score.tolist() and out.end_h.tolist() == ref.end_h.tolist()


# 2 * (16,287 + 64) = 32,702 of 32,703; 3 * 3 + 3 * (2 * 5,232 + 66) = 31,599 of 31,603.
@pytest.mark.parametrize("mode,scheme,length,packed", [(1, (2, -3, -3), 16287, True), (1, (2, -3, -3), 16288, False),
                                                       (0, (1, -1, -3), 5232, True), (0, (1, -1, -3), 5233, False)])
def test_warp16_value_range(engine, mode, scheme, length, packed):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    mt, mm, g = scheme
    rng = np.random.default_rng(length)
    h = rng.integers(0, 2, length).astype(np.uint8)
    H, V = [h, h], [h.copy(), (h ^ 2) if mode == 0 else np.roll(h, 5)]
    out = sg.align_codes(H, V, sg.Score(mt, mm, g), mode=mode, traceback=True, alphabet_size=4)
    assert bool(_kernels() & N.GBA_KERNEL_WARP16) == packed
    _same(out, sg.align_codes(H, V, sg.Score(mt, mm, g), mode=mode, traceback=True, alphabet_size=4,
                              flags=N.GBA_FLAG_NO_WARP16))


@pytest.mark.parametrize("m,n,scheme,warps", [(15, 7, (2, -1, -2), False), (42, 2, (2, -1, -2), True),
                                              (255, 255, (2, -1, -2), True), (256, 255, (2, -1, -2), False),
                                              (1000, 24, (2, -1, -2), True), (1000, 25, (2, -1, -2), False),
                                              (130, 125, (262, -60, -90), True), (130, 126, (262, -60, -90), False),
                                              (60, 50, (2, -1, 1), False), (60, 50, (-1, 2, -1), False)])
def test_enumerator(engine, m, n, scheme, warps):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    from seqan_gb300 import local_enum as LE
    rng = np.random.default_rng(m)
    H, V = _pairs(rng, m, n, 2)
    LE.local_enumerate(H, V, sg.Score(scheme[0], scheme[1], scheme[2], scheme[2]), 9 * abs(scheme[0]), 3, alphabet="dna5")
    assert bool(_kernels() & N.GBA_KERNEL_ENUM_WARP) == warps


@pytest.mark.parametrize("count,gap_open,paired", [(2000, -6, True), (200, -6, False), (2000, 0, False)])
def test_extension(engine, count, gap_open, paired):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    from seqan_gb300 import align_extend as X
    rng = np.random.default_rng(count)
    H, V = _pairs(rng, 60, 60, count)
    X.extend_alignments(H, V, [(25, 25, 30, 30)] * count, 3, sg.Score(2, -4, -1, gap_open), 20)
    assert bool(_kernels() & N.GBA_KERNEL_EXTEND2) == paired
