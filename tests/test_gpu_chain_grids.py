"""GPU parity of the chain kernel's grid fill where its shapes change, against the oracle: bands and
rectangles on both sides of 32 rows (where a lane's next column may begin before its last one ends),
grids of more than 32, 112 and 128 columns and traces beyond the shared memory kept for them, linear
and affine schemes, free ends."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _chain(rng, gap, seed, n_seeds, shift):
    """Seeds of `seed` residues, `gap` residues apart in H and gap + shift in V, alike on the seeds and
    mostly between them."""
    h, v, seeds = [], [], []
    nh = nv = 0
    for k in range(n_seeds + 1):
        g = rng.integers(0, 4, max(gap, 1)).astype(np.uint8)
        g2 = g.copy()
        g2[rng.random(len(g2)) < 0.2] = rng.integers(0, 4)
        g2 = np.concatenate([g2, rng.integers(0, 4, shift).astype(np.uint8)]) if shift else g2
        h.append(g); v.append(g2)
        nh += len(g); nv += len(g2)
        if k < n_seeds:
            s = rng.integers(0, 4, seed).astype(np.uint8)
            h.append(s); v.append(s)
            seeds.append((nh, nv, nh + seed, nv + seed))
            nh += seed; nv += seed
    return np.concatenate(h), np.concatenate(v), np.array(seeds, np.int32)


@pytest.mark.parametrize("k", [1, 7, 8, 15, 16, 40])
@pytest.mark.parametrize("scheme", [(2, -4, -1, -6), (2, -3, -5, -5)])
@pytest.mark.parametrize("fe", [0, 15])
def test_grid_shapes(engine, k, scheme, fe):
    import seqan_gb300 as sg
    from seqan_gb300.banded_chain import banded_chain_codes
    rng = np.random.default_rng(100 * k + fe)
    H, V, C = [], [], []
    for gap in (1, 3, 31, 33, 64, 150, 300):
        for seed in (1, 20, 33, 70, 140):
            h, v, c = _chain(rng, gap, seed, 3, (gap + seed) % 3)
            H.append(h); V.append(v); C.append(c)
    sc = sg.Score(scheme[0], scheme[1], scheme[2], scheme[3])
    cfg = sg.AlignConfig(bool(fe & 1), bool(fe & 2), bool(fe & 4), bool(fe & 8))
    score, status, ntr, segs = banded_chain_codes(H, V, C, sc, sc, cfg, k)
    for i in range(len(H)):
        o = O.oracle_banded_chain(H[i], V[i], C[i], scheme, scheme, fe, k)
        assert int(status[i]) == o.status, i
        if o.status == 0:
            assert (int(score[i]), int(ntr[i]), segs[i]) == (o.score, o.n_traces, o.segments), i
