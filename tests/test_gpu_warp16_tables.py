"""GPU parity of the packed 16-bit warp kernel with the 32-bit one on score tables whose entries lie far
below a byte and pairs whose best score is near the end of the 16-bit range: the step down from such a
score by one substitution is then as large as a half holds, in the columns past a pair's last one
too, and must not disturb the traceback bits of the cells that share its registers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAST = 4      # a letter of H's last column alone, which scores `low` against the others


def _table(match, low):
    t = np.full((5, 5), -3, np.int32)
    np.fill_diagonal(t, match)
    t[LAST, :LAST] = t[:LAST, LAST] = low
    return t


def _compare(H, V, table, mode, go, ge):
    import seqan_gb300 as sg
    from seqan_gb300 import _native as N
    score = sg.Score(0, 0, ge, go)
    score.matrix = np.ascontiguousarray(table)
    new = sg.align_codes(H, V, score, mode=mode, traceback=True, alphabet_size=5)
    kernels = sg.default_context().stats().dp_kernels
    old = sg.align_codes(H, V, score, mode=mode, traceback=True, alphabet_size=5, flags=N.GBA_FLAG_NO_WARP16)
    for f in ("score", "end_h", "end_v", "begin_h", "begin_v"):
        assert getattr(new, f).tolist() == getattr(old, f).tolist(), f
    assert [new.pair_segments(k) for k in range(len(H))] == [old.pair_segments(k) for k in range(len(H))]
    return kernels


def _pair(seed, match, n, insert):
    """V in H with `insert` residues more in the middle, then the letter that fits nothing."""
    rng = np.random.default_rng(seed)
    v = rng.integers(0, 4, n).astype(np.uint8)
    at = n // 2
    return np.concatenate([v[:at], rng.integers(0, 4, insert).astype(np.uint8), v[at:], [LAST]]).astype(np.uint8), v


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("low", [-128, -129, -650, -1000, -1024])
@pytest.mark.parametrize("match,n", [(2, 16240), (3, 10830), (14, 2267)])
def test_low_entries_near_the_range_end(engine, mode, match, low, n):
    """One pair and a few (bands on many warps): the columns past the last one, in every strip."""
    H, V = [], []
    for insert in (30, 7, 1):
        h, v = _pair(n + insert, match, n, insert)
        H.append(h)
        V.append(v)
    _compare(H[:1], V[:1], _table(match, low), mode, -2, -1)
    _compare(H, V, _table(match, low), mode, -2, -1)


@pytest.mark.parametrize("mode", [0, 1])
def test_long_pair(engine, mode):
    h, v = _pair(1, 1, 32500, 30)
    _compare([h], [v], _table(1, -1000), mode, -2, -1)


@pytest.mark.parametrize("tall", [False, True])
@pytest.mark.parametrize("short", [1, 2, 3, 5, 40])
def test_high_and_low_entries_near_the_lower_range_end(engine, short, tall):
    """Global scores near the lower end beside entries far above and below: a letter scores up to 400 or
    -1024 against the other sequence's letters."""
    rng = np.random.default_rng(short)
    t = rng.choice([300, -1024, -3], (5, 5)).astype(np.int32)
    H, V = [], []
    for _ in range(3):
        h = rng.integers(0, 5, short).astype(np.uint8)
        v = rng.integers(0, 5, 31380 - short).astype(np.uint8)
        H.append(h if tall else v)
        V.append(v if tall else h)
    _compare(H, V, t, 0, -2, -1)
