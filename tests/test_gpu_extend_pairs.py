"""GPU parity of the two-extensions-per-thread kernel of gba_extend_alignments with the oracle: sides
of sizes around its 16-row strips and 16-column tiles, odd counts, missing sides, X-drop terminators
from never to at once, linear and affine gaps, tables, scores at the edge of the 16-bit range, shared
sequences, several chunks' worth of sizes in one batch -- and batches just outside its rule."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65]
PAIRED_ROWS = 16        # tile_rows of a call that took the kernel


def _alignments(rng, count, sizes, letters, seed_len=3):
    """Alignments of which both sides take lengths from sizes; queries follow their databases."""
    H, V, pos = [], [], []
    for _ in range(count):
        a, b, c, d = (int(x) for x in rng.choice(sizes, 4))
        h = rng.integers(0, letters, a + seed_len + c).astype(np.uint8)
        v = rng.integers(0, letters, b + seed_len + d).astype(np.uint8)
        k = min(a, b)
        v[b - k:b] = h[a - k:a]                             # the left sides agree next to the seed
        k = min(c, d)
        v[b + seed_len:b + seed_len + k] = h[a + seed_len:a + seed_len + k]
        noise = rng.random(len(v)) < rng.choice([0.02, 0.15, 0.5])
        v[noise] = rng.integers(0, letters, int(noise.sum()))
        if rng.random() < 0.5 and len(v) > 12:              # a gap
            at, w = int(rng.integers(0, len(v) - 4)), int(rng.integers(1, 4))
            v = np.concatenate([v[:at], v[at + w:], v[at:at + w]])
        H.append(h)
        V.append(v)
        pos.append((a, b, a + seed_len, b + seed_len))
    return H, V, pos


def _check(pb, H, V, pos, direction=O.EXTEND_BOTH, paired=True, seed_h=None):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    from seqan_gb300 import align_extend as X
    score = (sg.Score(pb.match, pb.mismatch, pb.gap_extend, pb.gap_open) if pb.matrix is None
             else sg.Blosum62(pb.gap_extend, pb.gap_open))
    ctx = N.default_context()
    got = X.extend_alignments(H, V, pos, direction, score, pb.xdrop, seed_h=seed_h,
                              alphabet="dna5" if pb.matrix is None else "aa")
    if paired is not None:
        assert (ctx.stats().tile_rows == PAIRED_ROWS) == paired
    sides, hs, vs = [], [], []
    for k, (hb, vb, he, ve) in enumerate(pos):
        h, v = H[k if seed_h is None else seed_h[k]], V[k]
        if direction & O.EXTEND_LEFT and hb > 0 and vb > 0:
            sides.append((k, 0))
            hs.append(h[:hb][::-1].copy())
            vs.append(v[:vb][::-1].copy())
        if direction & O.EXTEND_RIGHT and he < len(h) and ve < len(v):
            sides.append((k, 1))
            hs.append(h[he:].copy())
            vs.append(v[ve:].copy())
    ref = O.oracle_batch(pb, hs, vs, traceback=True)
    seen = {}
    for t, (k, side) in enumerate(sides):
        segs = ref.segments[t] if side else O.reverse_partial_trace(ref.segments[t], pos[k][0], pos[k][1])
        seen[k, side] = (int(ref.score[t]), [tuple(int(x) for x in s) for s in segs])
    for k, e in enumerate(got):
        assert (e.left_score, e.left_segments) == seen.get((k, 0), (0, [])), k
        assert (e.right_score, e.right_segments) == seen.get((k, 1), (0, [])), k


@pytest.mark.parametrize("scheme", [(2, -4, -6, -1), (1, -2, -2, -2), (3, -2, -1, -4), (2, -1, -3, 0), (0, -1, -2, -1)])
@pytest.mark.parametrize("xdrop", [None, 1000, 25, 9, 1, 0, -5])
def test_sizes(engine, scheme, xdrop):
    rng = np.random.default_rng(100 * scheme[0] - 10 * scheme[3] + (xdrop or 3))
    H, V, pos = _alignments(rng, 2500, SIZES, 4)
    _check(O.Problem("extend", 0, None, *scheme, None, 32, "dna", xdrop), H, V, pos)


@pytest.mark.parametrize("direction", [O.EXTEND_LEFT, O.EXTEND_RIGHT])
def test_directions_and_missing_sides(engine, direction):
    rng = np.random.default_rng(7)
    H, V, pos = _alignments(rng, 5401, [1, 5, 16, 20, 40], 4)
    for k in range(0, len(pos), 5):        # seeds at a sequence's end: nothing to extend there
        a, b, c, d = pos[k]
        pos[k] = [(0, b, c, d), (a, 0, c, d), (a, b, len(H[k]), d), (a, b, c, len(V[k]))][(k // 5) % 4]
    pb = O.Problem("extend", 0, None, 2, -3, -5, -2, None, 32, "dna", 12)
    _check(pb, H, V, pos, direction)
    _check(pb, H, V, pos)


@pytest.mark.parametrize("gaps", [(-11, -1), (-9, -9)])
@pytest.mark.parametrize("xdrop", [None, 25])
def test_tables(engine, gaps, xdrop):
    from tests import golden_cases as G
    table = np.array(G.load("blosum62.json")["matrix"], dtype=np.int32)
    rng = np.random.default_rng(5)
    H, V, pos = _alignments(rng, 2300, SIZES, 27)
    _check(O.Problem("extend", 0, None, 0, 0, *gaps, table, 32, "aa", xdrop), H, V, pos)


@pytest.mark.parametrize("scheme", [(298, -1024, -180, -170), (-1, -1024, -170, -180), (298, 298, -150, -150)])
@pytest.mark.parametrize("xdrop", [None, 700])
def test_values_at_the_edge(engine, scheme, xdrop):
    """Sides of up to 45 residues: 298 * (45 + 64) and 170 * (90 + 66) lie just inside the rule."""
    rng = np.random.default_rng(3)
    H, V, pos = _alignments(rng, 2200, [1, 44, 45], 4)
    _check(O.Problem("extend", 0, None, *scheme, None, 32, "dna", xdrop), H, V, pos)


def test_uneven_sides_and_shared_database(engine):
    rng = np.random.default_rng(11)
    H, V, pos = _alignments(rng, 2400, [1, 3, 30, 100, 250, 300], 4)
    _check(O.Problem("extend", 0, None, 2, -4, -6, -1, None, 32, "dna", 20), H, V, pos, paired=None)
    H, V, pos = _alignments(rng, 300, [1, 3, 30, 60, 100], 4)
    _check(O.Problem("extend", 0, None, 2, -4, -6, -1, None, 32, "dna", 20), H, V, pos)
    h = rng.integers(0, 4, 300).astype(np.uint8)
    at = rng.integers(20, 270, 2500)
    V = [h[a - 20:a + 28].copy() for a in at]
    for v in V:
        v[rng.random(48) < 0.05] = 2
    pos = [(int(a), 20, int(a) + 8, 28) for a in at]
    _check(O.Problem("extend", 0, None, 1, -2, -4, -1, None, 32, "dna", 8), [h], V, pos,
           seed_h=np.zeros(len(pos), np.int32))


@pytest.mark.parametrize("scheme,sizes", [((2, -4, 0, -1), SIZES), ((2, -4, -3, 1), [1, 16, 20]), ((2, -4, 0, 0), [1, 16, 20]),
                                          ((1025, -4, -3, -2), [1, 16, 20]), ((300, -1024, -180, -170), [1, 46, 47]),
                                          ((2, -4, -6, -1), [1, 20, 1025])])
def test_outside_the_rule(engine, scheme, sizes):
    rng = np.random.default_rng(13)
    H, V, pos = _alignments(rng, 2200, sizes, 4)
    _check(O.Problem("extend", 0, None, *scheme, None, 32, "dna", 30), H, V, pos, paired=False)


def test_few_tall_sides_and_few_sides(engine):
    rng = np.random.default_rng(19)
    pb = O.Problem("extend", 0, None, 2, -4, -6, -1, None, 32, "dna", 30)
    _check(pb, *_alignments(rng, 400, [1, 20, 600], 4), paired=False)
    _check(pb, *_alignments(rng, 255, SIZES, 4), paired=False)


def test_several_trace_chunks(engine):
    """Sides of 250 residues whose traces exceed one chunk (4 GB), against batches of few sides."""
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    from seqan_gb300 import align_extend as X
    rng = np.random.default_rng(23)
    n, step = 70_000, 250
    H = rng.integers(0, 4, (n, 504)).astype(np.uint8)
    V = H.copy()
    noise = rng.random(V.shape) < 0.1
    V[noise] = rng.integers(0, 4, int(noise.sum()))
    V[:, 100:400] = np.where(np.arange(n)[:, None] % 3 == 0, V[:, 102:402], V[:, 100:400])
    H, V, pos = list(H), list(V), [(252, 252, 254, 254)] * n
    got = X.extend_alignments(H, V, pos, O.EXTEND_BOTH, sg.Score(2, -4, -1, -6), 40)
    assert N.default_context().stats().tile_rows == PAIRED_ROWS
    for at in [*range(0, n, 5000), n - step]:
        one = X.extend_alignments(H[at:at + step], V[at:at + step], pos[at:at + step], O.EXTEND_BOTH,
                                  sg.Score(2, -4, -1, -6), 40)
        assert N.default_context().stats().tile_rows != PAIRED_ROWS
        assert got[at:at + step] == one
