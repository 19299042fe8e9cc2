// traceback_kernels.cuh -- device traceback: trace matrix -> TraceSegment_ list -> CIGAR.
//
// One thread per pair walks back from the best cell exactly as the reference does:
//   start-cell correction          align/dp_algorithm_impl.h:1188-1205 (affine only)
//   initial direction              align/dp_traceback_impl.h:456-483 (PreferGapsAtEnd_ for affine)
//   tail / head gap segments       align/dp_traceback_impl.h:522-545 (global only; the
//                                  AlignExtend_ profile records the head only)
//   walk order and gap walkers     align/dp_traceback_impl.h:190-450 (GapsLeft)
//   segment recording              align/dp_trace_segment.h:318-337
// and writes the segments in the reference's order (traceback order).  Pairs of the warp layouts
// (dp_warp_kernels.cuh, dp_warp2_kernels.cuh) are walked by a whole warp instead
// (k_traceback_warp).  The CIGAR is the
// run-length form of the same alignment columns that getCigarString iterates
// (bam_io/cigar.h:261-339): DIAGONAL -> M, VERTICAL (gap in H) -> I, HORIZONTAL -> D, and a
// D run of at least 20 becomes N.
#pragma once

#include "dp_common.cuh"
#include "dp_banded2_kernels.cuh"
#include "dp_banded_kernels.cuh"
#include "dp_warp_kernels.cuh"
#include "dp_warp2_kernels.cuh"

namespace gba {

struct SegWriter {
    uint32_t *out;
    int cap;
    int n;
    bool leader;       // writes the records (all lanes of a warp walk keep the count)
    __device__ __forceinline__ void record(int hb, int vb, int len, int tv)
    {
        if (len == 0) return;
        uint32_t type;
        if (tv & TV_DIAG) type = TV_DIAG;
        else if (tv & TV_V) type = TV_V;
        else if (tv & TV_H) type = TV_H;
        else return;
        if (leader && n < cap) {
            uint32_t *o = out + 4 * int64_t(n);
            o[0] = uint32_t(hb);
            o[1] = uint32_t(vb);
            o[2] = uint32_t(len);
            o[3] = type;
        }
        ++n;
    }
};

// A walk's state: the current cell, its trace value and the length of the current fragment.
struct TraceWalk {
    int col, row, tv, frag;
};

// One lane's moves, one cell at a time; TAT(col, row) reads one trace byte.
template <typename Cell>
struct LaneSteps {
    Cell &TAT;
    __device__ __forceinline__ void diagonal(TraceWalk &w)
    {
        --w.col; --w.row; w.tv = TAT(w.col, w.row); ++w.frag;
    }
    // The reference's gap walkers (align/dp_traceback_impl.h:242-255, 320-332): through cells that
    // extend the gap, then one step more.  run: affine gaps (else the one step).
    __device__ __forceinline__ void vertical(TraceWalk &w, bool run)
    {
        if (run)
            while ((!(w.tv & TV_VO) || (w.tv & TV_V)) && w.row != 1) { --w.row; w.tv = TAT(w.col, w.row); ++w.frag; }
        --w.row; w.tv = TAT(w.col, w.row); ++w.frag;
    }
    __device__ __forceinline__ void horizontal(TraceWalk &w, bool run)
    {
        if (run)
            while ((!(w.tv & TV_HO) || (w.tv & TV_H)) && w.col != 1) { --w.col; w.tv = TAT(w.col, w.row); ++w.frag; }
        --w.col; w.tv = TAT(w.col, w.row); ++w.frag;
    }
};

// The same moves by a whole warp: the lanes read the next 32 cells in the walk's direction at once
// and a ballot finds where the run ends.  TAT.prefetch(col, row) asks for a cell's line.
template <typename Cell>
struct WarpSteps {
    Cell &TAT;
    int lane;
    __device__ __forceinline__ void diagonal(TraceWalk &w)
    {
        const int c = w.col - 1 - lane, r = w.row - 1 - lane;
        const int t = (c >= 0 && r >= 0) ? TAT(c, r) : int(TV_NONE);
        if (c > 64 && r > 64) TAT.prefetch(c - 64, r - 64);
        // the run ends at the first cell that does not continue it or lies on the border
        const uint32_t end = __ballot_sync(0xffffffffu, !(t & TV_DIAG) || c <= 0 || r <= 0);
        const int k = end ? __ffs(end) : 32;
        w.tv = __shfl_sync(0xffffffffu, t, k - 1);
        w.col -= k; w.row -= k; w.frag += k;
    }
    // One gap run along the rows (dr = 1) or the columns (dc = 1); ext / open: the direction's bits.
    __device__ __forceinline__ void gap(TraceWalk &w, bool run, int dc, int dr, int open, int ext)
    {
        auto goes_on = [&](int t, int at) { return (!(t & open) || (t & ext)) && at != 1; };
        for (;;) {
            const int c = w.col - dc * (lane + 1), r = w.row - dr * (lane + 1);
            const int t = (c >= 0 && r >= 0) ? TAT(c, r) : int(TV_NONE);
            // k cells of the run are passed, the (k + 1)-th move is the walker's last step
            int k = 0;
            if (run && goes_on(w.tv, dc ? w.col : w.row)) {
                const uint32_t stop = __ballot_sync(0xffffffffu, !goes_on(t, dc ? c : r));
                k = stop ? __ffs(stop) : 32;
            }
            const int moves = min(k + 1, 32);
            w.tv = __shfl_sync(0xffffffffu, t, moves - 1);
            w.col -= dc * moves; w.row -= dr * moves; w.frag += moves;
            if (k < 32) return;
        }
    }
    __device__ __forceinline__ void vertical(TraceWalk &w, bool run) { gap(w, run, 0, 1, TV_VO, TV_V); }
    __device__ __forceinline__ void horizontal(TraceWalk &w, bool run) { gap(w, run, 1, 0, TV_HO, TV_H); }
};

// Walks pair p back from its best cell; TAT(col, row) reads one trace byte.  With leader false
// the walk only counts (the other lanes of a warp walk).
template <typename Cell, typename Steps>
__device__ __forceinline__ void traceback_pair(const TraceArgs &a, int p, Cell &TAT, Steps &steps, bool leader)
{
    const PairDesc d = a.pairs[p];
    const int m = d.m, n = d.n;
    int col = a.end_h[p], row = a.end_v[p];
    const bool affine = a.affine != 0;
    const bool global = a.local == 0;

    SegWriter w;
    w.out = a.seg_slots + 4 * a.seg_slot_off[p];
    w.cap = int(a.seg_slot_off[p + 1] - a.seg_slot_off[p]);
    w.n = 0;
    w.leader = leader;

    int tv = TAT(col, row);
    if (affine) {
        const int s = a.score[p];
        if (a.best_f[p] == s) { tv &= ~TV_DIAG; tv |= TV_MFV; }
        else if (a.best_e[p] == s) { tv &= ~TV_DIAG; tv |= TV_MFH; }
    } else if (a.dynamic) {
        // DynamicGaps: the best cell's flags (vertical first) decide
        // (align/dp_algorithm_impl.h:1235-1249).
        const int fl = a.best_e[p];
        if (fl & 1) { tv &= ~TV_DIAG; tv |= TV_MFV; }
        else if (fl & 2) { tv &= ~TV_DIAG; tv |= TV_MFH; }
    }
    int last;
    if (affine) {
        if (tv & TV_MFV) { tv &= (TV_V | TV_VO | TV_MFV); last = TV_V; }
        else if (tv & TV_MFH) { tv &= (TV_H | TV_HO | TV_MFH); last = TV_H; }
        else last = TV_DIAG;
    } else {
        if (tv & TV_DIAG) last = TV_DIAG;
        else if (tv & (TV_V | TV_MFV)) last = TV_V;
        else if (tv & (TV_H | TV_MFH)) last = TV_H;
        else last = TV_NONE;
    }
    if (global && !a.extend) {
        if (row != n) w.record(m, row, n - row, TV_V);
        if (col != m) w.record(col, row, m - col, TV_H);
    }
    TraceWalk wk{col, row, tv, 0};
    auto turn = [&](int dir) {
        if (!(last & dir)) { w.record(wk.col, wk.row, wk.frag, last); last = dir; wk.frag = 0; }
    };
    // Every move goes left or up, so the walk ends after at most m + n cells.
    while (!(wk.col <= 0 || wk.row <= 0) && wk.tv != TV_NONE) {
        if (wk.tv & TV_DIAG) {
            turn(TV_DIAG);
            steps.diagonal(wk);
        } else if ((wk.tv & TV_MFV) && (wk.tv & (TV_V | TV_VO))) {
            turn(TV_V);
            steps.vertical(wk, affine && (wk.tv & TV_V));
        } else if ((wk.tv & TV_MFH) && (wk.tv & (TV_H | TV_HO))) {
            turn(TV_H);
            steps.horizontal(wk, affine && (wk.tv & TV_H));
        } else {
            break;
        }
    }
    col = wk.col;
    row = wk.row;
    w.record(col, row, wk.frag, last);
    if (global) {
        if (row != 0) w.record(0, 0, row, TV_V);
        if (col != 0) w.record(0, 0, col, TV_H);
    }
    if (!leader) return;
    a.seg_count[p] = w.n;
    if (w.n > 0 && w.n <= w.cap) {
        const uint32_t *lastSeg = w.out + 4 * int64_t(w.n - 1);
        a.begin_h[p] = int32_t(lastSeg[0]);
        a.begin_v[p] = int32_t(lastSeg[1]);
    } else {
        a.begin_h[p] = 0;
        a.begin_v[p] = 0;
    }

    // CIGAR: walk the segments in alignment order (reverse of the list).
    if (a.cigar_slots && w.n <= w.cap) {
        uint32_t *co = a.cigar_slots + a.cigar_slot_off[p];
        const int ccap = int(a.cigar_slot_off[p + 1] - a.cigar_slot_off[p]);
        int nc = 0;
        int curOp = -1;
        uint32_t curLen = 0;
        for (int k = w.n - 1; k >= -1; --k) {
            int op = -1;
            uint32_t len = 0;
            if (k >= 0) {
                const uint32_t *sg = w.out + 4 * int64_t(k);
                len = sg[2];
                op = sg[3] == TV_DIAG ? 0 : (sg[3] == TV_V ? 1 : 2);  // M, I, D
            }
            if (op != curOp) {
                if (curLen > 0) {
                    int emit = (curOp == 2 && curLen >= 20) ? 3 : curOp;  // N
                    if (nc < ccap) co[nc] = (curLen << 4) | uint32_t(emit);
                    ++nc;
                }
                curOp = op;
                curLen = 0;
            }
            curLen += len;
        }
        a.cigar_count[p] = nc;
    } else if (a.cigar_slots) {
        a.cigar_count[p] = 0;
    }
}

// One thread per pair: the one-pair-per-thread layouts (strips, bands).
__global__ void __launch_bounds__(128) k_traceback(TraceArgs a)
{
    const int64_t slot = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (slot >= a.num_slots) return;
    const int p = a.order[slot];
    if (p < 0) return;   // padding slot
    const PairDesc d = a.pairs[p];
    const int m = d.m;
    const uint8_t *T = a.trace + d.trace_off;
    const int bw = a.band_w, bu = a.band_upper;
    const bool affine = a.affine != 0;
    auto TAT = [&](int c, int r) -> int {
        if (bw && d.rows)   // two pairs a thread
            return int(trace_at_band2(T, int((d.trace_off >> 4) & 31), d.rows - 1, bw, bu, affine, c, r));
        return bw ? int(trace_at_band(T, d.trace_off, bw, bu, affine, c, r)) : int(trace_at(T, m, c, r));
    };
    LaneSteps<decltype(TAT)> steps{TAT};
    traceback_pair(a, p, TAT, steps, true);
}

// Trace readers of the two warp layouts.
template <int R>
struct WarpCell {
    const uint8_t *T;
    int m, n;
    __device__ __forceinline__ int operator()(int c, int r) const { return T[trace_off_warp(m, n, R, c, r)]; }
    __device__ __forceinline__ void prefetch(int c, int r) const
    {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(T + trace_off_warp(m, n, R, c, r)));
    }
};
struct Warp2Cell {
    const uint8_t *T;
    int m, rows;
    bool local, affine;
    __device__ __forceinline__ int operator()(int c, int r) const { return w2_trace_at(T, m, rows, local, affine, c, r); }
    __device__ __forceinline__ void prefetch(int c, int r) const
    {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(T + w2_trace_off(m, rows, local, c, r)));
    }
};

// One warp per pair.  A walk is a chain of dependent reads of the trace, each a trip to L2 or HBM
// (0.4-0.9 us), and the paths are mostly diagonal runs, so the lanes read the next 32 cells of the
// run at once and a ballot finds its end: one trip per run of up to 32 cells instead of one per
// cell.  Lines 64 cells ahead on the diagonal are asked for early (a gap shifts the walk by one row
// or column, which mostly stays in those lines).  Measured, whole calls with tracebacks: 8 pairs of
// 10,000 bp 6.58 -> 5.09 ms, 2,000 pairs of 100 to 10,000 bp 11.5 -> 8.9 ms, 20,000 protein pairs
// 5.88 -> 5.02 ms (before: one thread per pair, or a warp per long pair reading a 16 KB tile of the
// trace into shared memory and walking it cell by cell).
template <bool W2, int R>
__global__ void __launch_bounds__(128) k_traceback_warp(TraceArgs a)
{
    const int64_t slot = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (slot >= a.num_slots) return;
    const int p = a.order[slot];
    if (p < 0) return;   // padding slot
    const PairDesc d = a.pairs[p];
    const int lane = threadIdx.x & 31;
    if (W2) {
        Warp2Cell cell{a.trace + d.trace_off, d.m, d.rows, a.local != 0, a.affine != 0};
        WarpSteps<Warp2Cell> steps{cell, lane};
        traceback_pair(a, p, cell, steps, lane == 0);
    } else {
        WarpCell<R> cell{a.trace + d.trace_off, d.m, d.n};
        WarpSteps<WarpCell<R>> steps{cell, lane};
        traceback_pair(a, p, cell, steps, lane == 0);
    }
}

// Packs per-pair slot outputs densely: dst[off[k] ..] = src[slot_off[k] .. + count[k]].
__global__ void k_compact_u32(const uint32_t *src, const int64_t *slot_off, const int32_t *count,
                              const int64_t *dense_off, uint32_t *dst, int64_t num_pairs, int words)
{
    const int64_t p = int64_t(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x / 32);
    if (p >= num_pairs) return;
    const int lane = threadIdx.x & 31;
    const int64_t cnt = int64_t(count[p]) * words;
    const uint32_t *s = src + slot_off[p] * words;
    uint32_t *d = dst + dense_off[p] * words;
    for (int64_t i = lane; i < cnt; i += 32) d[i] = s[i];
}

}  // namespace gba
