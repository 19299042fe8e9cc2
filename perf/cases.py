"""Performance cases of the engine: what is timed, through the C-ABI that a user's program calls.

A case is a dict of plain values; its "kind" names one of the engine's paths and the other values
are that path's sizes and options.  listed() holds one case of each path at the size its users run
it at, draw() gives further cases of the same paths over their whole range.  prepare() makes the
inputs from a seed (and the plan that such a program keeps), run() is one pass, work() what the
pass cannot do without.  All outputs are whole numbers, equal from run to run; a packed list
(segments, CIGAR words) comes back as its buffer, which holds zeros behind the list's end.

Host calls take and fill page-locked host buffers, as a program that feeds batches keeps them;
device-resident calls take and fill device memory.
"""
import ctypes as C
import math

import numpy as np
import torch

from seqan_gb300 import _native as N
from seqan_gb300.scoring import BLOSUM62_AA27
from seqan_gb300.workloads import AA20_CODES, load_background

# Integer operations per cell of each recurrence.
OPS = {"linear_global": 5, "linear_local": 6, "affine_global": 9, "affine_local": 10}
SEED_LEN = 19
SCORES = N.GBA_OUT_SCORE | N.GBA_OUT_END


# ------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # A small call: a thousand unrelated 150 bp pairs, linear gaps, 32-bit scores.  Latency of
        # one call and few warps in flight.
        {"name": "dna_linear_1k", "kind": "small", "pairs": 1024, "lo": 150, "hi": 150, "affine": False,
         "traceback": False, "related": False},
        # The headline batch: overlap scoring of uneven 100-300 bp reads, affine gaps, on codes
        # that lie in device memory, with the plan kept.
        {"name": "dna_affine_100k", "kind": "scores", "pairs": 100_000, "lo": 100, "hi": 300},
        # Protein search: one query against a database, best local scores.
        {"name": "protein_search_20k", "kind": "search", "query": 350, "pairs": 20_000, "median": 300},
        # Protein pairs aligned locally with their tracebacks.
        {"name": "protein_local_20k", "kind": "protein", "pairs": 20_000, "median": 300, "related": 0.3},
        # Read verification in a mapper: reads of one length against the windows of their
        # candidate places, banded, CIGARs; every batch has the same shape, so the plan is kept.
        {"name": "reads_banded_1m", "kind": "reads", "pairs": 1_000_000, "read": 150, "flank": 10, "half": 16},
        # A service's batch: mostly short pairs, some of thousands, 1% of 10,000 bp, tracebacks.
        {"name": "dna_mixed_2k", "kind": "mixed", "pairs": 2000},
        # A few long pairs: each alone must spread over the device.
        {"name": "dna_long_8", "kind": "long", "pairs": 8, "length": 10_000, "traceback": True},
        # Seed extension in a mapper: X-drop on reads and windows in device memory.
        {"name": "xdrop_reads_1m", "kind": "xdrop", "seeds": 1_000_000, "read": 150, "flank": 50, "drop": 20},
        # Alignment extension around seeds in both directions, with X-drop.
        {"name": "extend_reads_250k", "kind": "extend", "seeds": 250_000, "read": 150, "flank": 50, "drop": 20},
        # Genomic pairs aligned around chains of anchors.
        {"name": "banded_chain_10k", "kind": "chain", "pairs": 10_000, "lo": 1000, "hi": 3000, "extension": 15},
        # Suboptimal local alignments: up to ten of each pair.
        {"name": "suboptimal_10k", "kind": "enumerate", "pairs": 10_000, "lo": 100, "hi": 200, "count": 10, "half": 0},
        # Reading a sequencing run: a FASTA text into codes and offsets.
        {"name": "fasta_reads_2m", "kind": "fasta", "records": 2_000_000, "lo": 150, "hi": 150, "width": 80},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "scores", "search", "protein", "reads", "mixed", "long", "xdrop", "extend", "chain",
                       "enumerate", "fasta"])
    if kind == "small":
        lo = rng.randint(30, 200)
        return {"kind": kind, "pairs": _log(rng, 8, 4000), "lo": lo, "hi": lo + rng.choice([0, rng.randint(1, 150)]),
                "affine": rng.random() < 0.6, "traceback": rng.random() < 0.5, "related": rng.random() < 0.6}
    if kind == "scores":
        lo = rng.randint(40, 250)
        return {"kind": kind, "pairs": _log(rng, 5000, 200_000), "lo": lo, "hi": lo + rng.randint(0, 250)}
    if kind == "search":
        return {"kind": kind, "query": _log(rng, 60, 1000), "pairs": _log(rng, 1000, 40_000),
                "median": rng.randint(150, 400)}
    if kind == "protein":
        return {"kind": kind, "pairs": _log(rng, 1000, 30_000), "median": rng.randint(120, 400),
                "related": round(rng.uniform(0.1, 0.9), 2)}
    if kind == "reads":
        return {"kind": kind, "pairs": _log(rng, 50_000, 1_000_000), "read": rng.randint(75, 251),
                "flank": rng.randint(8, 14), "half": rng.randint(6, 24)}
    if kind == "mixed":
        return {"kind": kind, "pairs": _log(rng, 100, 3000)}
    if kind == "long":
        return {"kind": kind, "pairs": rng.randint(1, 16), "length": _log(rng, 3000, 15_000),
                "traceback": rng.random() < 0.6}
    if kind in ("xdrop", "extend"):
        top = 1_000_000 if kind == "xdrop" else 250_000
        return {"kind": kind, "seeds": _log(rng, top // 20, top), "read": rng.randint(75, 251),
                "flank": rng.randint(20, 60), "drop": rng.randint(10, 30)}
    if kind == "chain":
        lo = rng.randint(400, 2000)
        return {"kind": kind, "pairs": _log(rng, 500, 8000), "lo": lo, "hi": lo + rng.randint(100, 1500),
                "extension": rng.randint(5, 25)}
    if kind == "enumerate":
        lo = rng.randint(50, 150)
        return {"kind": kind, "pairs": _log(rng, 500, 8000), "lo": lo, "hi": lo + rng.randint(0, 80),
                "count": rng.randint(1, 10), "half": rng.choice([0, rng.randint(8, 24)])}
    lo = rng.randint(36, 200)
    return {"kind": kind, "records": _log(rng, 50_000, 1_500_000), "lo": lo, "hi": lo + rng.choice([0, 101]),
            "width": rng.choice([60, 70, 80])}


# ------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------
class Rand:
    """Seeded draws in device memory."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 7919 + 12345)

    def ints(self, lo, hi, shape, dtype=torch.uint8):
        return torch.randint(lo, hi, shape if isinstance(shape, tuple) else (int(shape),), generator=self.g,
                             device="cuda", dtype=dtype)

    def unit(self, shape):
        return torch.rand(shape if isinstance(shape, tuple) else (int(shape),), generator=self.g, device="cuda")


def _offsets(lengths):
    off = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=off[1:])
    return off


def _mutated(r, h, off, subs, indels):
    """The sequences with substitutions and single-base insertions and deletions: codes, offsets,
    and each residue's place in the result (-1: deleted) with whether it stayed as it was."""
    n = h.numel()
    u = r.unit(n)
    kept, ins = u >= indels / 2, (u >= indels / 2) & (u < indels)
    u = r.unit(n)
    sub = u < subs
    base = torch.where(sub, (h + r.ints(1, 4, n)) % 4, h)
    width = kept.to(torch.int64) + ins.to(torch.int64)
    end = torch.cumsum(width, 0)
    place = end - width + ins
    v = r.ints(0, 4, int(end[-1]))
    v[place[kept]] = base[kept]
    ends = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), end])
    return v, ends[off], torch.where(kept, place, torch.full_like(place, -1)), kept & ~sub


def _host(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _room(n, dtype=torch.int32):
    return torch.zeros(n if isinstance(n, tuple) else (int(n),), dtype=dtype, pin_memory=True)


def _dna_pairs(r, lengths, related, subs=0.05, indels=0.01):
    off = _offsets(lengths)
    h = r.ints(0, 4, int(off[-1]))
    if related:
        v, ov, _, _ = _mutated(r, h, off, subs, indels)
    else:
        v, ov = r.ints(0, 4, h.numel()), off.clone()
    return h, off, v, ov


def _residues(r, n):
    """Amino-acid codes in the proportions of natural proteins."""
    p = torch.tensor(np.cumsum(load_background()), dtype=torch.float32, device="cuda")
    codes = torch.tensor(np.array(AA20_CODES), dtype=torch.uint8, device="cuda")
    return codes[torch.searchsorted(p, r.unit(n)).clamp(max=19)]


def _protein_lengths(r, n, median):
    z = torch.randn(n, generator=r.g, device="cuda")
    return torch.exp(math.log(median) + 0.5 * z).round().clamp(50, 1000).to(torch.int64)


def _reads(r, n, length, flank, subs, indels):
    """Reads of one length from a random 10 Mbp genome, the windows around their origins, where in
    its window each read base comes from and whether it equals that base there."""
    genome = r.ints(0, 4, 10_000_000)
    span = length + 2 * flank
    origin = r.ints(flank, genome.numel() - span, n, torch.int64)
    windows = genome[(origin - flank)[:, None] + torch.arange(span, device="cuda")]
    u = r.unit((n, length))
    ins = u < indels / 2
    dele = (u >= indels / 2) & (u < indels)
    at = torch.arange(length, device="cuda") + torch.cumsum(dele, 1) - torch.cumsum(ins, 1) + flank
    at.clamp_(0, span - 1)
    reads = torch.gather(windows, 1, at)
    sub = r.unit((n, length)) < subs
    reads = torch.where(sub, (reads + r.ints(1, 4, (n, length))) % 4, reads)
    reads = torch.where(ins, r.ints(0, 4, (n, length)), reads)
    return windows, reads, at, ~sub & ~ins


def _read_seeds(r, windows, reads, at, same):
    """One exact SEED_LEN-mer of each read on its own diagonal (any place where it has none), as
    Seed<Simple> rows."""
    n, length = reads.shape
    k = SEED_LEN
    steps = torch.zeros((n, length), dtype=torch.int32, device="cuda")
    steps[:, 1:] = (same[:, 1:] & same[:, :-1] & (at[:, 1:] == at[:, :-1] + 1)).to(torch.int32)
    run = torch.cumsum(steps, 1)
    good = (run[:, k - 1:] - run[:, :length - k + 1]) == k - 1
    start = (r.unit((n, length - k + 1)) * (good.to(torch.float32) + 1e-3)).argmax(1)
    h = torch.gather(at, 1, start[:, None])[:, 0].clamp(max=windows.shape[1] - k)
    d = h - start
    return torch.stack([h, start, h + k, start + k, d, d], 1)


# ------------------------------------------------------------------------------------------
# Calls
# ------------------------------------------------------------------------------------------
def _p(t):
    return C.c_void_p(t.data_ptr())


def _align_params(c, mode=N.GBA_GLOBAL, linear=False, bits=16, outputs=SCORES, protein=False, free=0, band=None):
    p = N.GbaParams()
    p.mode, p.free_ends, p.score_bits, p.outputs = mode, free, bits, outputs
    if protein:
        p.gap_open, p.gap_extend, p.alphabet_size = -11, -1, 27
        p.matrix = BLOSUM62_AA27.ctypes.data_as(C.c_void_p)
    elif linear:
        p.match, p.mismatch, p.gap_open, p.gap_extend, p.alphabet_size = 2, -3, -5, -5, 4
    else:
        p.match, p.mismatch, p.gap_open, p.gap_extend, p.alphabet_size = 2, -4, -6, -1, 4
    if band:
        p.band_on, p.band_lower, p.band_upper = 1, band[0], band[1]
    return p


class Plan:
    """A gba_plan that goes with its owner."""

    def __init__(self, ctx, params, batch):
        self.ctx, self.handle = ctx, C.c_void_p()
        ctx.check(N.lib().gba_plan_create(ctx.handle, C.byref(params), C.byref(batch), C.byref(self.handle)), "plan")

    def __del__(self):
        N.lib().gba_plan_destroy(self.ctx.handle, self.handle)


def _traced(s, n, room):
    """Result buffers of a call with tracebacks, `room` segments in all."""
    s["segments"], s["segment_offsets"] = _room((room, 4)), _room(n + 1, torch.int64)
    s["begin_h"], s["begin_v"] = _room(n), _room(n)
    r = s["result"]
    r.begin_h, r.begin_v, r.segment_offsets = _p(s["begin_h"]), _p(s["begin_v"]), _p(s["segment_offsets"])
    r.segments, r.segment_capacity = _p(s["segments"]), room


def _host_batch(s, h, oh, v, ov, params, traceback, room, shared=False):
    n = ov.numel() - 1
    s["h"], s["oh"], s["v"], s["ov"] = (_host(t) for t in (h, oh, v, ov))
    s["score"], s["end_h"], s["end_v"], s["status"] = (_room(n) for _ in range(4))
    s["params"], s["result"] = params, N.GbaResult()
    s["batch"] = N.GbaBatch(n, _p(s["h"]), _p(s["oh"]), _p(s["v"]), _p(s["ov"]), 1 if shared else 0, 0)
    r = s["result"]
    r.score, r.end_h, r.end_v, r.pair_status = (_p(s[k]) for k in ("score", "end_h", "end_v", "status"))
    if traceback:
        _traced(s, n, room)
    return s


def _room_for(case, n):
    """Segments to make room for: the same for every seed, above what the path's inputs give."""
    kind = case["kind"]
    if kind == "small":
        return n * (2 * case["hi"] + 64) if not case["related"] else n * (case["hi"] // 4 + 32)
    if kind == "protein":
        return n * (case["median"] // 3 + 32)
    if kind == "mixed":
        return n * 150 + 10_000
    if kind == "long":
        return n * (case["length"] // 8 + 64)
    return n * (case["hi"] // 8 + 32)


def _traceback_bits(on):
    return SCORES | (N.GBA_OUT_SEGMENTS if on else 0)


def prepare(case, seed):
    r, ctx = Rand(seed), N.default_context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx}
    if kind == "small":
        n = case["pairs"]
        h, oh, v, ov = _dna_pairs(r, r.ints(case["lo"], case["hi"] + 1, n, torch.int64), case["related"])
        p = _align_params(case, linear=not case["affine"], bits=16 if case["affine"] else 32,
                          outputs=_traceback_bits(case["traceback"]))
        return _host_batch(s, h, oh, v, ov, p, case["traceback"], _room_for(case, n))
    if kind == "scores":
        n = case["pairs"]
        h, oh, v, ov = _dna_pairs(r, r.ints(case["lo"], case["hi"] + 1, n, torch.int64), True)
        s["h"], s["v"] = h, v
        s["score"], s["end_h"], s["end_v"] = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
        oh, ov = oh.cpu(), ov.cpu()
        s["plan"] = Plan(ctx, _align_params(case), N.GbaBatch(n, _p(h), _p(oh), _p(v), _p(ov), 0, 0))
        s["batch"], s["result"] = N.GbaBatch(n, _p(h), None, _p(v), None, 0, 0), N.GbaResult()
        s["result"].score, s["result"].end_h, s["result"].end_v = _p(s["score"]), _p(s["end_h"]), _p(s["end_v"])
        return s
    if kind == "search":
        lengths = _protein_lengths(r, case["pairs"], case["median"])
        ov = _offsets(lengths)
        q = _residues(r, case["query"])
        oh = torch.tensor([0, case["query"]], dtype=torch.int64)
        p = _align_params(case, mode=N.GBA_LOCAL, protein=True)
        return _host_batch(s, q, oh, _residues(r, int(ov[-1])), ov, p, False, 0, shared=True)
    if kind == "protein":
        n = case["pairs"]
        lh, lv = _protein_lengths(r, n, case["median"]), _protein_lengths(r, n, case["median"])
        kin = r.unit(n) < case["related"]
        lv = torch.where(kin, lh, lv)
        oh, ov = _offsets(lh), _offsets(lv)
        h, v = _residues(r, int(oh[-1])), _residues(r, int(ov[-1]))
        pair = torch.repeat_interleave(torch.arange(n, device="cuda"), lv)
        take = kin[pair] & (r.unit(v.numel()) < 0.4)
        source = oh[pair] + torch.arange(v.numel(), device="cuda") - ov[pair]
        v[take] = h[source[take]]
        p = _align_params(case, mode=N.GBA_LOCAL, protein=True, outputs=_traceback_bits(True))
        return _host_batch(s, h, oh, v, ov, p, True, _room_for(case, n))
    if kind == "reads":
        n, length, flank = case["pairs"], case["read"], case["flank"]
        windows, reads, _, _ = _reads(r, n, length, flank, 0.02, 0.002)
        s["h"], s["v"] = windows, reads
        oh = torch.arange(n + 1, dtype=torch.int64) * windows.shape[1]
        ov = torch.arange(n + 1, dtype=torch.int64) * length
        s["score"], s["end_h"], s["end_v"] = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
        p = _align_params(case, outputs=_traceback_bits(True) | N.GBA_OUT_CIGAR, free=N.GBA_FREE_TOP | N.GBA_FREE_BOTTOM,
                          band=(flank - case["half"], flank + case["half"]))
        s["plan"] = Plan(ctx, p, N.GbaBatch(n, _p(windows), _p(oh), _p(reads), _p(ov), 0, 0))
        s["batch"] = N.GbaBatch(n, _p(windows), None, _p(reads), None, 0, 0)
        s["device"], s["result"] = N.GbaResult(), N.GbaResult()
        s["device"].score, s["device"].end_h, s["device"].end_v = _p(s["score"]), _p(s["end_h"]), _p(s["end_v"])
        _traced(s, n, 6 * n)
        s["cigar"], s["cigar_offsets"] = _room(6 * n), _room(n + 1, torch.int64)
        s["result"].cigar, s["result"].cigar_capacity = _p(s["cigar"]), 6 * n
        s["result"].cigar_offsets = _p(s["cigar_offsets"])
        return s
    if kind in ("mixed", "long"):
        n = case["pairs"]
        if kind == "mixed":
            u = r.unit(n)
            lengths = torch.where(u < 0.90, r.ints(100, 501, n, torch.int64),
                                  torch.where(u < 0.99, r.ints(1000, 5001, n, torch.int64),
                                              torch.full((n,), 10_000, dtype=torch.int64, device="cuda")))
        else:
            lengths = r.ints(case["length"] * 9 // 10, case["length"] + 1, n, torch.int64)
        traceback = case.get("traceback", True)
        h, oh, v, ov = _dna_pairs(r, lengths, True)
        p = _align_params(case, outputs=_traceback_bits(traceback))
        return _host_batch(s, h, oh, v, ov, p, traceback, _room_for(case, n))
    if kind in ("xdrop", "extend"):
        n = case["seeds"]
        windows, reads, at, same = _reads(r, n, case["read"], case["flank"], 0.03, 0.003)
        seeds = _read_seeds(r, windows, reads, at, same)
        oh = torch.arange(n + 1, dtype=torch.int64, device="cuda") * windows.shape[1]
        ov = torch.arange(n + 1, dtype=torch.int64, device="cuda") * case["read"]
        host = kind == "extend"
        s["h"], s["v"], s["oh"], s["ov"], s["seeds"] = ((_host(t) if host else t.contiguous())
                                                        for t in (windows, reads, oh, ov, seeds))
        s["batch"] = N.GbaSeedBatch(n, _p(s["h"]), _p(s["oh"]), n, _p(s["v"]), _p(s["ov"]), n, None, None,
                                    case["read"])
        if not host:
            s["params"] = N.GbaExtendParams(N.GBA_GAPPED_XDROP, N.GBA_EXTEND_BOTH, case["drop"], 1, -2, -2, None, 0, 0)
            s["grown"] = torch.empty_like(s["seeds"])
            s["scores"] = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
            return s
        s["params"] = N.GbaExtendAlignParams(N.GBA_EXTEND_BOTH, 1, case["drop"], 2, -4, -6, -1, None, 0, 0, 0, 0)
        s["left"], s["right"], s["segment_offsets"] = _room(n), _room(n), _room(2 * n + 1, torch.int64)
        s["segments"] = _room((12 * n, 4))
        s["result"] = N.GbaExtendAlignResult(_p(s["left"]), _p(s["right"]), _p(s["segments"]), 12 * n,
                                             _p(s["segment_offsets"]))
        return s
    if kind == "chain":
        return _prepare_chain(s, case, r)
    if kind == "enumerate":
        n, count = case["pairs"], case["count"]
        lengths = r.ints(case["lo"], case["hi"] + 1, n, torch.int64)
        oh = _offsets(lengths)
        h = r.ints(0, 4, int(oh[-1]))
        v, ov, _, _ = _mutated(r, h, oh, 0.1, 0.02)
        other = torch.repeat_interleave(torch.arange(n, device="cuda") % 2 == 0, ov[1:] - ov[:-1])
        v = torch.where(other, r.ints(0, 4, v.numel()), v)   # every other pair is unrelated
        s["h"], s["oh"], s["v"], s["ov"] = (_host(t) for t in (h, oh, v, ov))
        s["batch"] = N.GbaBatch(n, _p(s["h"]), _p(s["oh"]), _p(s["v"]), _p(s["ov"]), 0, 0)
        s["params"] = N.GbaEnumParams(2, -1, -2, 10, None, 0, count)
        s["band"] = case["half"]
        s["count"], s["status"], s["segment_offsets"] = _room(n), _room(n), _room(n * count + 1, torch.int64)
        s["each"] = [_room((n, count)) for _ in range(5)]
        room = n * count * 40
        s["segments"] = _room((room, 4))
        s["result"] = N.GbaEnumResult(_p(s["count"]), _p(s["status"]), *(_p(t) for t in s["each"]), _p(s["segments"]),
                                      room, _p(s["segment_offsets"]))
        return s
    return _prepare_fasta(s, case, r)


def _prepare_chain(s, case, r):
    n = case["pairs"]
    lengths = r.ints(case["lo"], case["hi"] + 1, n, torch.int64)
    oh = _offsets(lengths)
    h = r.ints(0, 4, int(oh[-1]))
    v, ov, place, same = _mutated(r, h, oh, 0.05, 0.01)
    pair = torch.repeat_interleave(torch.arange(n, device="cuda"), lengths)
    # Anchors: the runs of at least 20 equal residues along the alignment, at most 64 of a pair.
    go = same[1:] & same[:-1] & (place[1:] == place[:-1] + 1) & (pair[1:] == pair[:-1])
    no = torch.zeros(1, dtype=torch.bool, device="cuda")
    first = torch.nonzero(same & ~torch.cat([no, go]))[:, 0]
    last = torch.nonzero(same & ~torch.cat([go, no]))[:, 0]
    long = last - first >= 19
    first, last = first[long], last[long]
    owner = pair[first]
    found = torch.bincount(owner, minlength=n)
    rank = torch.arange(first.numel(), device="cuda") - _offsets(found)[owner]
    of = found[owner]
    pick = (of <= 64) | ((rank * 64) // of != ((rank - 1) * 64) // of)
    first, last, owner = first[pick], last[pick], owner[pick]
    begin_h, begin_v, size = first - oh[owner], place[first] - ov[owner], last - first + 1
    seeds = torch.stack([begin_h, begin_v, begin_h + size, begin_v + size], 1).to(torch.int32)
    so = _offsets(torch.bincount(owner, minlength=n))
    s["h"], s["oh"], s["v"], s["ov"], s["seeds"], s["so"] = (_host(t) for t in (h, oh, v, ov, seeds, so))
    scheme = N.GbaSimpleScore(2, -4, -1, -6)
    s["params"] = N.GbaChainParams(scheme, scheme, 0, case["extension"], 0)
    s["batch"] = N.GbaBatch(n, _p(s["h"]), _p(s["oh"]), _p(s["v"]), _p(s["ov"]), 0, 0)
    s["chains"] = N.GbaChainSeeds(_p(s["seeds"]), _p(s["so"]))
    s["score"], s["status"], s["traces"] = (_room(n) for _ in range(3))
    room = _room_for(case, n)
    s["segments"], s["segment_offsets"] = _room((room, 4)), _room(n + 1, torch.int64)
    s["result"] = N.GbaChainResult(_p(s["score"]), _p(s["status"]), _p(s["traces"]), _p(s["segments"]), room,
                                   _p(s["segment_offsets"]))
    return s


def _prepare_fasta(s, case, r):
    n, width = case["records"], case["width"]
    lengths = r.ints(case["lo"], case["hi"] + 1, n, torch.int64)
    head = torch.tensor(list(b">read"), dtype=torch.uint8, device="cuda")
    digits = 8
    first = head.numel() + digits + 1                       # header line with its line end
    start = _offsets(first + lengths + (lengths + width - 1) // width)
    text = torch.full((int(start[-1]),), 10, dtype=torch.uint8, device="cuda")
    text[start[:-1, None] + torch.arange(head.numel(), device="cuda")] = head
    tens = 10 ** torch.arange(digits - 1, -1, -1, device="cuda")
    name = (torch.arange(n, device="cuda")[:, None] // tens % 10 + 48).to(torch.uint8)
    text[start[:-1, None] + head.numel() + torch.arange(digits, device="cuda")] = name
    off = _offsets(lengths)
    total = int(off[-1])
    letters = torch.tensor(list(b"ACGTNacgtn"), dtype=torch.uint8, device="cuda")
    code = r.ints(0, 4, total)
    code[r.unit(total) < 0.001] = 4
    code[r.unit(total) < 0.03] += 5                         # lower case
    j = torch.arange(total, device="cuda") - torch.repeat_interleave(off[:-1], lengths)
    at = torch.repeat_interleave(start[:-1] + first, lengths) + j + j // width
    text[at] = letters[code.to(torch.int64)]
    s["text"] = _host(text)
    s["codes"] = _room(n * case["hi"], torch.uint8)
    s["id_begin"], s["id_end"], s["seq_off"] = (_room(n + 1, torch.int64) for _ in range(3))
    s["records"] = N.GbaSeqRecords(n + 1, n * case["hi"], _p(s["id_begin"]), _p(s["id_end"]), _p(s["seq_off"]), None,
                                   _p(s["codes"]), None, 0, 0, -1)
    return s


def run(s):
    L, ctx, kind = N.lib(), s["ctx"], s["kind"]
    if kind == "scores":
        ctx.check(L.gba_plan_execute(ctx.handle, s["plan"].handle, C.byref(s["batch"]), C.byref(s["result"])), kind)
        return [s["score"], s["end_h"], s["end_v"]]
    if kind == "reads":
        ctx.check(L.gba_plan_execute(ctx.handle, s["plan"].handle, C.byref(s["batch"]), C.byref(s["device"])), kind)
        ctx.check(L.gba_plan_fetch(ctx.handle, s["plan"].handle, C.byref(s["result"])), kind)
        return [s["score"], s["end_h"], s["end_v"], s["begin_h"], s["begin_v"], s["segment_offsets"],
                s["segments"], s["cigar_offsets"], s["cigar"]]
    if kind == "xdrop":
        # The seeds grow in place: a copy on this program's stream, complete before the engine's.
        s["grown"].copy_(s["seeds"])
        torch.cuda.current_stream().synchronize()
        ctx.check(L.gba_extend_seeds_device(ctx.handle, C.byref(s["params"]), C.byref(s["batch"]), _p(s["grown"]),
                                            _p(s["scores"])), kind)
        ctx.check(L.gba_synchronize(ctx.handle), kind)      # reports seeds outside their sequences
        return [s["grown"], s["scores"]]
    if kind == "extend":
        ctx.check(L.gba_extend_alignments(ctx.handle, C.byref(s["params"]), C.byref(s["batch"]), _p(s["seeds"]),
                                          C.byref(s["result"])), kind)
        return [s["left"], s["right"], s["segment_offsets"], s["segments"]]
    if kind == "chain":
        ctx.check(L.gba_banded_chain(ctx.handle, C.byref(s["params"]), C.byref(s["batch"]), C.byref(s["chains"]),
                                     C.byref(s["result"])), kind)
        return [s["score"], s["status"], s["traces"], s["segment_offsets"], s["segments"]]
    if kind == "enumerate":
        if s["band"]:
            ctx.check(L.gba_local_enumerate_banded(ctx.handle, C.byref(s["params"]), -s["band"], s["band"],
                                                   C.byref(s["batch"]), C.byref(s["result"])), kind)
        else:
            ctx.check(L.gba_local_enumerate(ctx.handle, C.byref(s["params"]), C.byref(s["batch"]),
                                            C.byref(s["result"])), kind)
        have = torch.arange(s["each"][0].shape[1])[None, :] < s["count"][:, None]
        return [s["count"], s["status"], s["segment_offsets"], s["segments"]] + \
            [torch.where(have, t, 0) for t in s["each"]]
    if kind == "fasta":
        rec = s["records"]
        ctx.check(L.gba_read_fasta(ctx.handle, _p(s["text"]), s["text"].numel(), 5, C.byref(rec)), kind)
        n = int(rec.num)
        return [s["id_begin"][:n], s["id_end"][:n], s["seq_off"][:n + 1], s["codes"]]
    ctx.check(L.gba_align_batch(ctx.handle, C.byref(s["params"]), C.byref(s["batch"]), C.byref(s["result"])), kind)
    out = [s["score"], s["end_h"], s["end_v"], s["status"]]
    if "segments" in s:
        out += [s["begin_h"], s["begin_v"], s["segment_offsets"], s["segments"]]
    return out


# ------------------------------------------------------------------------------------------
# What a pass cannot do without, from the expected sizes
# ------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("small", "scores"):
        n, lo, hi = case["pairs"], case["lo"], case["hi"]
        mean = (lo + hi) / 2
        square = mean * mean + (hi - lo) * (hi - lo + 2) / 12
        out = 12 + (8 + 8 + 16 * 6 if case.get("traceback") else 0) + (4 if kind == "small" else 0)
        return {"bytes": n * (2 * mean + 16 + out),
                "flops": n * square * OPS["affine_global" if case.get("affine", True) else "linear_global"]}
    if kind in ("search", "protein"):
        n, mean = case["pairs"], case["median"] * 1.12          # log-normal, clipped
        if kind == "search":
            return {"bytes": n * (mean + 8 + 16), "flops": n * mean * case["query"] * OPS["affine_local"]}
        return {"bytes": n * (2 * mean + 16 + 32 + 16 * 6),
                "flops": n * mean * mean * (1 + 0.23 * case["related"]) * OPS["affine_local"]}
    if kind == "reads":
        n, length = case["pairs"], case["read"]
        return {"bytes": n * (2 * length + 2 * case["flank"] + 36 + 20 * 2),
                "flops": n * length * (2 * case["half"] + 1) * OPS["affine_global"]}
    if kind == "mixed":
        n = case["pairs"]
        mean, square = 0.9 * 300 + 0.09 * 3000 + 0.01 * 1e4, 0.9 * 103e3 + 0.09 * 10.3e6 + 0.01 * 1e8
        return {"bytes": n * (2 * mean + 52 + 16 * 13), "flops": n * square * OPS["affine_global"]}
    if kind == "long":
        n, length = case["pairs"], case["length"] * 0.95
        out = length * 0.02 * 16 if case["traceback"] else 0
        return {"bytes": n * (2 * length + 32 + out), "flops": n * length * length * OPS["affine_global"]}
    if kind in ("xdrop", "extend"):
        n, length, flank = case["seeds"], case["read"], case["flank"]
        rest = length - SEED_LEN
        if kind == "xdrop":
            return {"bytes": n * (2 * length + 2 * flank + 16 + 96 + 8), "flops": n * 2 * rest * case["drop"] * 0.47 * 6}
        cells = 0.78 * 2 * (rest * rest / 3 + flank * rest / 2)
        return {"bytes": n * (2 * length + 2 * flank + 16 + 48 + 24 + 16 * 4), "flops": n * cells * OPS["affine_global"]}
    if kind == "chain":
        n, mean = case["pairs"], (case["lo"] + case["hi"]) / 2
        return {"bytes": n * mean * (2 + 16 * 0.02 + 16 * 0.02), "flops": n * mean * 7.5 * case["extension"] *
                OPS["affine_global"]}
    if kind == "enumerate":
        n, lo, hi = case["pairs"], case["lo"], case["hi"]
        mean = (lo + hi) / 2
        cells = mean * (2 * case["half"] + 1) if case["half"] else mean * mean + (hi - lo) * (hi - lo + 2) / 12
        return {"bytes": n * (2 * mean + 24 + case["count"] * (20 + 8 + 16 * 6)), "flops": n * cells * OPS["linear_local"]}
    n, mean = case["records"], (case["lo"] + case["hi"]) / 2
    return {"bytes": n * (14 + mean + mean / case["width"] + mean + 24), "flops": 0}
