"""The banded chain kernel with its lanes out of step, on the CPU (tests/cpp/chain_lanes.cpp): between two
warp-wide operations the lanes run one after another, first to last, last to first and in random
orders.  Every order has to give the oracle's chains: no lane may rely on another being at the same
instruction."""
import shutil
import struct
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O

SOURCE = Path(__file__).parent / "cpp" / "chain_lanes.cpp"


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("lanes")
    flags = ["g++", "-std=c++17", "-O1", "-g", "-w"]
    subprocess.check_call(flags + ["-DCHAIN_PLAN", "-c", str(SOURCE), "-o", str(d / "plan.o")])
    subprocess.check_call(flags + ["-c", str(SOURCE), "-o", str(d / "lanes.o")])
    subprocess.check_call(["g++", str(d / "plan.o"), str(d / "lanes.o"), "-o", str(d / "lanes")])
    return str(d / "lanes")


def _chain(rng, gap, seed, count, shift):
    """`count` seeds of `seed` residues, about `gap` residues apart, mostly alike between them."""
    h, v, seeds = [], [], []
    nh = nv = 0
    for k in range(count + 1):
        g = rng.integers(0, 4, max(gap, 1)).astype(np.uint8)
        g2 = g.copy()
        g2[rng.random(len(g2)) < 0.2] = rng.integers(0, 4)
        g2 = np.concatenate([g2, rng.integers(0, 4, shift).astype(np.uint8)])
        h.append(g)
        v.append(g2)
        nh += len(g)
        nv += len(g2)
        if k < count:
            s = rng.integers(0, 4, seed).astype(np.uint8)
            h.append(s)
            v.append(s)
            seeds.append((nh, nv, nh + seed, nv + seed))
            nh += seed
            nv += seed
    return np.concatenate(h), np.concatenate(v), np.array(seeds, np.int32)


def _run(program, problems, scheme, gap_scheme, fe, k, order):
    data = b""
    affine = int(scheme[2] != scheme[3] or gap_scheme[2] != gap_scheme[3])
    for h, v, seeds in problems:
        data += struct.pack("<15i", len(h), len(v), len(seeds), *scheme, *gap_scheme, fe, k, affine, 32)
        data += h.tobytes() + v.tobytes() + np.ascontiguousarray(seeds, np.int32).tobytes()
    out = subprocess.run([program, str(order)], input=data, capture_output=True, timeout=300)
    assert out.returncode == 0, out.returncode
    got, at = [], 0
    for _ in problems:
        met, status, score, traces, count = struct.unpack_from("<5i", out.stdout, at)
        at += 20
        segs = [tuple(int(x) for x in s) for s in np.frombuffer(out.stdout, np.uint32, 4 * count, at).reshape(-1, 4)]
        at += 16 * count
        got.append((met, status, score, traces, segs))
    return got


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("scheme,gap_scheme", [((2, -4, -1, -6), (2, -4, -1, -6)), ((2, -3, -5, -5), (1, -1, -1, -1))])
@pytest.mark.parametrize("fe,k", [(0, 4), (15, 4), (0, 15)])
def test_lanes_in_any_order(program, order, scheme, gap_scheme, fe, k):
    rng = np.random.default_rng(100 * k + fe)
    problems = [_chain(rng, gap, seed, count, (gap + seed) % 3)
                for gap, seed, count in [(1, 1, 1), (1, 20, 1), (3, 9, 2), (12, 10, 4), (40, 33, 3), (150, 70, 2)]]
    problems.append((problems[3][0], problems[3][1], problems[3][2][:0]))   # no seed
    problems.append((problems[3][0][:9], problems[3][1], problems[3][2]))   # seeds beyond the sequence
    got = _run(program, problems, scheme, gap_scheme, fe, k, order)
    for i, (h, v, seeds) in enumerate(problems):
        ref = O.oracle_banded_chain(h, v, seeds, scheme, gap_scheme, fe, k)
        assert got[i][0] == 1, i
        assert got[i][1] == ref.status, i
        if ref.status == 0:
            assert got[i][2:] == (ref.score, ref.n_traces, ref.segments), i
