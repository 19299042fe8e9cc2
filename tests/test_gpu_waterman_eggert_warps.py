"""GPU parity of the warp-per-pair Waterman-Eggert enumerator with the oracle at its edges: sequences
around the 32-column and 32-row steps, heaps around the levels where a word of its bits begins (32
and 1,024 nodes), every cell pushed
(cutoffs at and below zero), many ties (match 1), free and costly gaps, few letters, the largest
matrix, trace and score it takes -- and batches just outside its rule."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _key(a):
    return (a.score, a.row0, a.row1, a.h_begin, a.h_end, a.v_begin, a.v_end)


def _check(H, V, scheme, cutoff, count, step=1):
    import seqan_gb300 as sg
    from seqan_gb300 import local_enum as LE
    match, mismatch, gap = scheme
    got = LE.local_enumerate(H, V, sg.Score(match, mismatch, gap, gap), cutoff, count, alphabet="dna5")
    for k in range(0, len(H), step):
        ref = O.oracle_local_enumerate(H[k], V[k], match, mismatch, gap, cutoff, max_count=count)
        undefined = bool(ref) and ref[-1] is None
        ref = ref[:-1] if undefined else ref
        assert got[k].undefined_next == undefined, k
        assert [_key(a) for a in got[k].alignments] == [_key(a) for a in ref], k
        assert [a.segments for a in got[k].alignments] == [a.segments for a in ref], k


def _pairs(rng, sizes, count, letters, related=0.5):
    from seqan_gb300 import workloads as W
    H, V = [], []
    for _ in range(count):
        h = rng.integers(0, letters, int(rng.choice(sizes))).astype(np.uint8)
        n = int(rng.choice(sizes))
        v = rng.integers(0, letters, n).astype(np.uint8)
        if rng.random() < related:
            w = W.mutate(rng, h, 0.1, 0.04)[:n]
            v[:len(w)] = w
        H.append(h)
        V.append(v)
    return H, V


SIZES = [1, 2, 21, 22, 23, 24, 31, 32, 33, 63, 64, 65, 96, 97]


@pytest.mark.parametrize("scheme", [(2, -1, -2), (1, -1, -1), (1, 0, 0), (5, -4, -9), (2, 1, -1), (0, 2, -1)])
@pytest.mark.parametrize("cutoff", [-3, 0, 1, 7, 20])
@pytest.mark.parametrize("letters", [1, 2, 4])
def test_sizes_and_ties(engine, scheme, cutoff, letters):
    rng = np.random.default_rng(1000 * letters + 10 * cutoff + scheme[0])
    H, V = _pairs(rng, SIZES, 60, letters)
    _check(H, V, scheme, cutoff, 14)


def test_empty_sequences_and_one_pair(engine):
    rng = np.random.default_rng(2)
    H, V = _pairs(rng, SIZES, 20, 4)
    H[3], V[5], H[7], V[7] = H[3][:0], V[5][:0], H[7][:0], V[7][:0]
    _check(H, V, (2, -1, -2), 5, 5)
    _check(H[:1], V[:1], (2, -1, -2), 5, 50)


@pytest.mark.parametrize("lengths,scheme,cutoff", [
    ((255, 255), (2, -1, -2), 0),          # 2^16 cells, all of them in the heap
    ((255, 255), (2, -1, -2), 30),
    ((1000, 24), (2, -1, -2), 12),         # 1,024 steps
    ((24, 1000), (2, -1, -2), 12),
    ((130, 125), (262, -60, -90), 900),    # 262 * 125 = 32,750
    ((256, 255), (2, -1, -2), 30),         # outside: cells, steps, scores, gaps and matches that pay / cost
    ((1000, 25), (2, -1, -2), 12),
    ((130, 126), (262, -60, -90), 900),
    ((60, 50), (2, -1, 1), 5),
    ((60, 50), (-1, 2, -1), 5),
])
def test_edges_of_the_rule(engine, lengths, scheme, cutoff):
    from seqan_gb300 import workloads as W
    rng = np.random.default_rng(lengths[0] + scheme[0])
    H, V = [], []
    for k in range(4):
        h = rng.integers(0, 4, lengths[0]).astype(np.uint8)
        v = rng.integers(0, 4, lengths[1]).astype(np.uint8)
        if k % 2:
            w = W.mutate(rng, h, 0.08, 0.02)[:lengths[1]]
            v[:len(w)] = w
        H.append(h)
        V.append(v)
    _check(H, V, scheme, cutoff, 6)


def test_more_pairs_than_resident_warps(engine):
    rng = np.random.default_rng(9)
    H, V = _pairs(rng, [20, 40, 60, 80], 9000, 4)
    _check(H, V, (2, -1, -2), 10, 4, step=9)
