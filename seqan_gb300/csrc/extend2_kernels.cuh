// extend2_kernels.cuh -- the AlignExtend_ DP of extendAlignment, two extensions per thread.
//
// For batches large enough to fill the device this way, of sides whose values fit 16 bits
// (ext_paired in extend_host.cuh): each thread runs two extensions of about the same size in the two
// 16-bit halves of its registers (biased values and trace bit planes as in dp_warp2_kernels.cuh),
// and the trace is written in the same pass that finds the best cell and the last column.
//
// Columns go in tiles of kX2Cols, and a tile's rows in strips of kX2Rows held in registers; a strip
// hands its bottom row (S, F) and the column maxima so far down through shared memory, and its
// column state (S, E) to the next tile through a per-warp scratch.  The terminator of
// align_extend/dp_scout_xdrop.h looks at whole columns, so it is applied to the tile's column maxima
// when the tile is done, column by column as the reference does: the columns past the one it stops
// at (half a tile on average) are computed for nothing and nothing reads their trace.  The scout's
// row is the first one holding its column's maximum; it is looked for only in columns whose maximum
// beats everything before them.
//
// With gap scores below 0 the best cell never ends in a gap (a cell of an earlier column, or higher
// up in the column, would score more), so its E and F are not kept: the start-cell correction of
// the traceback (align/dp_algorithm_impl.h:1188-1205) never applies.
//
// Bound by the ALU pipe (80% busy; about 14 instructions per two cells go there).  250,000 read
// seeds (150 bp in 250 bp windows, both sides, 2/-4/-6/-1, X-drop 20, 3.4 G cells) take 2.4 ms, the
// traceback 0.12; the column-synchronous form (extend_kernels.cuh: a group of lanes per extension,
// a scan over the lanes for the vertical gaps, a score pass and a trace pass) takes 29.6 and 0.5,
// most of it instructions between the lanes.  16 rows are what 128 registers (four blocks an SM) hold
// of S, E and codes; score tables need more, at three blocks.
#pragma once

#include "dp_common.cuh"
#include "extend_kernels.cuh"
#include "packed16.cuh"

namespace gba {

constexpr int kX2Rows = 16, kX2Cols = 16;
constexpr int kX2Inf = -31680;

struct X2Seed { int64_t begin_h, begin_v, end_h, end_v, lower, upper; };

// A side's result, by id = 2 * alignment + side (0 left, 1 right).
struct X2Out {
    int32_t score, col, row, last;
};

struct X2Args {
    const uint8_t *seq_h, *seq_v;
    const int64_t *off_h, *off_v;
    const int32_t *seed_h, *seed_v;   // null: alignment k lies on sequences k
    const X2Seed *seeds;
    const int32_t *order;             // 64 ids per warp: the low halves, then the high halves; -1: none
    const int32_t *cols;              // per warp: the most columns of its sides
    const int64_t *trace_off;         // per warp
    int32_t num_warps;
    int32_t *next;                    // work counter
    int32_t match, mismatch, gap_open, gap_extend;
    const int32_t *matrix;
    int32_t asize;
    int32_t xdrop_on, xdrop;
    uint8_t *trace;
    uint2 *state;                     // per resident warp: state_rows x 32 (S, E)
    int32_t state_rows;               // a multiple of kX2Rows
    X2Out *out;
    unsigned long long *cells;
};

struct X2Task {
    const uint8_t *h, *v;             // residue j (1-based) at h[hs * j]
    int32_t m, n, step;
};

__device__ __forceinline__ X2Task x2_task(const X2Args &a, int id)
{
    const int k = id >> 1;
    const int hi = a.seed_h ? a.seed_h[k] : k, vi = a.seed_v ? a.seed_v[k] : k;
    const X2Seed s = a.seeds[k];
    const uint8_t *h = a.seq_h + a.off_h[hi], *v = a.seq_v + a.off_v[vi];
    if (id & 1)
        return X2Task{h + s.end_h - 1, v + s.end_v - 1, int32_t(a.off_h[hi + 1] - a.off_h[hi] - s.end_h),
                      int32_t(a.off_v[vi + 1] - a.off_v[vi] - s.end_v), 1};
    return X2Task{h + s.begin_h, v + s.begin_v, int32_t(s.begin_h), int32_t(s.begin_v), -1};
}

// Byte offset in a warp's trace of the 16-byte chunk of (col, strip) of a lane: words (D, V) of rows
// 0-7 and 8-15, then (X, Y); row r of the strip is bit r % 8 of bytes 0 / 1 (low / high half) and 2 / 3.
__host__ __device__ inline int64_t x2_chunk(int cols, int col, int strip, int lane)
{
    return ((int64_t(strip) * cols + col - 1) * 32 + lane) * 16;
}
__host__ __device__ inline int64_t x2_trace_bytes(int cols, int n)
{
    return int64_t((n + kX2Rows - 1) / kX2Rows) * cols * 512;
}

__device__ __forceinline__ uint32_t x2_both(int x) { return pack2(x + 0x8000, x + 0x8000); }
__device__ __forceinline__ int x2_half(uint32_t x, int h) { return int(h ? x >> 16 : x & 0xffffu) - 0x8000; }
__device__ __forceinline__ uint32_t x2_max(uint32_t a, uint32_t b) { return __vimax3_u16x2(a, b, b); }
__device__ __forceinline__ uint32_t x2_equal(uint32_t small, uint32_t large) { return small - large + 0x80008000u; }
__device__ __forceinline__ uint32_t x2_signs(uint32_t a, uint32_t b) { return prmt(a, b, 0xFDB9); }

// Per column of the tile: the row above the next strip (S, F), the column's maximum and the row that
// first holds it where that may matter.
struct X2Shared {
    uint4 col[kX2Cols][128];
    uint32_t codes[kX2Cols][128];
};

template <bool AFFINE, bool MATRIX>
__global__ void __launch_bounds__(128, MATRIX ? 3 : 4) k_extend2(X2Args a)
{
    __shared__ X2Shared sh;
    __shared__ int smat[MATRIX ? 32 * 32 : 1];
    if (MATRIX) {
        for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
            const int r = i >> 5, c = i & 31;
            smat[i] = (r < a.asize && c < a.asize) ? a.matrix[r * a.asize + c] : 0;
        }
        __syncthreads();
    }
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + tid) >> 5;
    uint2 *const state = a.state + warp * a.state_rows * 32 + lane;
    const int open = AFFINE ? a.gap_open : a.gap_extend, ext = a.gap_extend, edge = max(open, ext);
    const uint32_t OPEN2 = pack2(open, open), EXTL = uint32_t(ext) * 0x00010001u;
    const uint32_t MATCHL = uint32_t(a.match) * 0x00010001u;
    const uint32_t MISS = uint32_t(a.match) - uint32_t(a.mismatch);      // what a mismatch costs against a match
    const uint32_t INF2 = x2_both(kX2Inf);
    // S of a border cell at distance i from the origin
    auto border = [&](int i) { return i == 0 ? 0 : open + (i - 1) * edge; };
    unsigned long long cells = 0;

    for (;;) {
        int w = 0;
        if (lane == 0) w = atomicAdd(a.next, 1);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= a.num_warps) break;
        const int idA = a.order[int64_t(w) * 64 + lane], idB = a.order[int64_t(w) * 64 + 32 + lane];
        const int cols = a.cols[w];
        uint8_t *const T = a.trace + a.trace_off[w];
        if (idA >= 0) {
            const X2Task A = x2_task(a, idA);
            X2Task B = A;
            if (idB >= 0) B = x2_task(a, idB);
            const int mh[2] = {A.m, idB >= 0 ? B.m : 0}, nh[2] = {A.n, idB >= 0 ? B.n : 0};
            const int M = max(mh[0], mh[1]), N = max(nh[0], nh[1]);
            // column 0
            for (int i = 1; i <= (N + kX2Rows - 1) / kX2Rows * kX2Rows; ++i)
                state[(i - 1) * 32] = make_uint2(x2_both(border(i)), INF2);
            int best[2] = {0, 0}, bestC[2] = {0, 0}, bestR[2] = {0, 0}, last[2] = {mh[0], mh[1]};
            bool flag[2] = {a.xdrop_on && 0 >= a.xdrop, a.xdrop_on && 0 >= a.xdrop};
            bool done[2] = {false, idB < 0};
            for (int c0 = 1; c0 <= M && !(done[0] && done[1]); c0 += kX2Cols) {
                const int nc = min(kX2Cols, M - c0 + 1);
                for (int c = 0; c < nc; ++c) {
                    const int j = c0 + c;
                    const uint32_t s = x2_both(border(j));
                    sh.col[c][tid] = make_uint4(s, INF2, s, 0);          // row 0
                    const uint32_t x = j <= mh[0] ? A.h[A.step * j] : 0u, y = j <= mh[1] ? B.h[B.step * j] : 0u;
                    sh.codes[c][tid] = x * 0x101u | (y * 0x101u) << 16;
                }
                uint32_t diagTop = x2_both(border(c0 - 1));              // S(row above the strip, c0 - 1)
                const uint32_t before = pack2(best[0] + 0x8000, best[1] + 0x8000);
                for (int i0 = 0; i0 < N; i0 += kX2Rows) {
                    uint32_t S[kX2Rows], E[kX2Rows], vc[kX2Rows];
#pragma unroll
                    for (int r = 0; r < kX2Rows; ++r) {
                        const int i = i0 + r + 1;
                        const uint2 q = state[(i - 1) * 32];
                        S[r] = q.x;
                        E[r] = q.y;
                        const uint32_t x = i <= nh[0] ? A.v[A.step * i] : 0u, y = i <= nh[1] ? B.v[B.step * i] : 0u;
                        vc[r] = x * 0x101u | (y * 0x101u) << 16;
                    }
                    const bool partial = i0 + kX2Rows > nh[0] || i0 + kX2Rows > nh[1];
                    uint32_t diagNext = diagTop;
                    diagTop = S[kX2Rows - 1];
                    uint32_t run = before;                               // maxima of the columns before this one
                    uint8_t *tr = T + x2_chunk(cols, c0, i0 / kX2Rows, lane);
#pragma unroll 1
                    for (int c = 0; c < nc; ++c, tr += 512) {
                        const uint4 q = sh.col[c][tid];
                        const uint32_t hc = sh.codes[c][tid];
                        uint32_t up = q.x, upF = q.y, diag = diagNext;
                        diagNext = up;
                        uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
#pragma unroll
                        for (int r = 0; r < kX2Rows; ++r) {
                            uint32_t inter;
                            if (MATRIX) {
                                const uint32_t sb = pack2(smat[(hc & 31u) << 5 | (vc[r] & 31u)],
                                                          smat[(hc >> 16 & 31u) << 5 | (vc[r] >> 16 & 31u)]);
                                inter = __viaddmax_u16x2(diag, sb, 0u);
                            } else {
                                // 1 in the halves whose codes differ
                                inter = diag + MATCHL - __vimin3_u16x2(hc ^ vc[r], 0x00010001u, 0x00010001u) * MISS;
                            }
                            diag = S[r];
                            uint32_t e, f, eExt = 0, fExt = 0;
                            if (AFFINE) {
                                eExt = E[r] + EXTL;
                                e = __viaddmax_u16x2(S[r], OPEN2, eExt);
                                fExt = upF + EXTL;
                                f = __viaddmax_u16x2(up, OPEN2, fExt);
                            } else {
                                e = S[r] + EXTL;
                                f = up + EXTL;
                            }
                            const uint32_t g = x2_max(e, f), s = x2_max(inter, g);
                            const uint32_t bit = 0x01010101u << (r & 7);
                            const uint32_t dv = x2_signs(x2_equal(inter, s), x2_equal(f, g)) & bit;
                            const uint32_t xy = AFFINE ? x2_signs(x2_equal(eExt, e), x2_equal(fExt, f)) & bit : 0u;
                            if (r < 8) { w0 |= dv; w2 |= xy; } else { w1 |= dv; w3 |= xy; }
                            S[r] = s;
                            E[r] = e;
                            up = s;
                            upF = f;
                        }
                        *reinterpret_cast<uint4 *>(tr) = make_uint4(w0, w1, w2, w3);
                        // the column's maximum over the rows inside the matrix
                        auto inside = [&](int r) {
                            return (i0 + r < nh[0] ? 0x0000ffffu : 0u) | (i0 + r < nh[1] ? 0xffff0000u : 0u);
                        };
                        uint32_t mx;
                        if (partial) {
                            mx = S[0] & inside(0);
#pragma unroll
                            for (int r = 1; r < kX2Rows; ++r) mx = x2_max(mx, S[r] & inside(r));
                        } else {
                            mx = S[0];
#pragma unroll
                            for (int r = 1; r + 1 < kX2Rows; r += 2) mx = __vimax3_u16x2(mx, S[r], S[r + 1]);
                            mx = x2_max(mx, S[kX2Rows - 1]);
                        }
                        const uint32_t top = x2_max(q.z, run);
                        uint32_t row = q.w;
                        if (x2_max(mx, top) != top) {
                            uint32_t first = 0;
#pragma unroll
                            for (int r = kX2Rows - 1; r >= 0; --r) {
                                const uint32_t eq = __vcmpeq2(S[r], mx) & inside(r);
                                first = (first & ~eq) | (uint32_t(i0 + r + 1) * 0x00010001u & eq);
                            }
                            const uint32_t more = __vcmpgtu2(mx, q.z);
                            row = (row & ~more) | (first & more);
                        }
                        const uint32_t colmax = x2_max(mx, q.z);
                        run = x2_max(run, colmax);
                        sh.col[c][tid] = make_uint4(up, upF, colmax, row);
                    }
#pragma unroll
                    for (int r = 0; r < kX2Rows; ++r) state[(i0 + r) * 32] = make_uint2(S[r], E[r]);
                }
                // the scout and the terminator, column by column
                for (int c = 0; c < nc; ++c) {
                    const int j = c0 + c;
                    const uint4 q = sh.col[c][tid];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (done[h] || j > mh[h]) continue;
                        const int cm = x2_half(q.z, h);
                        if (cm > best[h]) {
                            best[h] = cm;
                            bestC[h] = j;
                            bestR[h] = int(h ? q.w >> 16 : q.w & 0xffffu);
                        }
                        if (a.xdrop_on && best[h] - cm >= a.xdrop) flag[h] = true;
                        if (j == mh[h]) done[h] = true;
                        else if (flag[h]) {
                            done[h] = true;
                            last[h] = j;
                        }
                    }
                }
            }
            a.out[idA] = X2Out{best[0], bestC[0], bestR[0], last[0]};
            cells += (unsigned long long)(last[0] + 1) * (nh[0] + 1);
            if (idB >= 0) {
                a.out[idB] = X2Out{best[1], bestC[1], bestR[1], last[1]};
                cells += (unsigned long long)(last[1] + 1) * (nh[1] + 1);
            }
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) cells += __shfl_down_sync(0xffffffffu, cells, o);
    if (lane == 0 && cells) atomicAdd(a.cells, cells);
}

// Traceback of each side from its best cell to the origin (the walk of k_extend_traceback), one thread
// per side in the order of the DP; segments to slots of seg_cap[warp] each, counts by id.
template <bool AFFINE>
__global__ void __launch_bounds__(128) k_extend2_traceback(X2Args a, const int64_t *seg_off, const int32_t *seg_cap,
                                                           ExtSegment *segs, int64_t *slot, int32_t *count)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t w = t >> 6;
    if (w >= a.num_warps) return;
    const int id = a.order[t];
    if (id < 0) return;
    const int half = int(t >> 5) & 1, lane = int(t & 31), cols = a.cols[w];
    const X2Out o = a.out[id];
    const uint8_t *T = a.trace + a.trace_off[w];
    const int cap = seg_cap[w];
    const int64_t at = seg_off[w] + (t & 63) * cap;
    ExtSegment *s = segs + at;
    auto word = [&](int col, int row, int plane) {
        const int strip = (row - 1) / kX2Rows, r = (row - 1) % kX2Rows;
        const uint32_t *q = reinterpret_cast<const uint32_t *>(T + x2_chunk(cols, col, strip, lane));
        return q[plane + (r >> 3)] >> (8 * half + (r & 7));
    };
    int cnt = 0, col = o.col, row = o.row, frag = 0;
    // Cells are read when the walk stands on them; on row or column 0 it is over.
    int last = XT_DIAG;
    auto turn = [&](int dir) {
        if (last != dir) {
            ext_record(s, cap, cnt, col, row, frag, last);
            last = dir;
            frag = 0;
        }
    };
    while (col > 0 && row > 0) {
        const uint32_t dv = word(col, row, 0);
        if (dv & 1u) {
            turn(XT_DIAG);
            --col; --row; ++frag;
        } else if ((dv >> 16) & 1u) {
            turn(XT_V);
            // through cells whose F extends, then one step more; linear gaps go step by step
            if (AFFINE)
                while (((word(col, row, 2) >> 16) & 1u) && row != 1) { --row; ++frag; }
            --row; ++frag;
        } else {
            turn(XT_H);
            if (AFFINE)
                while ((word(col, row, 2) & 1u) && col != 1) { --col; ++frag; }
            --col; ++frag;
        }
    }
    ext_record(s, cap, cnt, col, row, frag, last);
    // TraceHead_ (align/dp_traceback_impl.h:538-545)
    if (row != 0) ext_record(s, cap, cnt, 0, 0, row, XT_V);
    if (col != 0) ext_record(s, cap, cnt, 0, 0, col, XT_H);
    slot[id] = at;
    count[id] = cnt > cap ? 0 : cnt;   // (cap holds every walk)
}

// Each side's segments to the packed result and its score, one thread per id; the left side's are
// mapped back from the reversed prefixes (_reversePartialTrace: begin = length - end, order reversed).
__global__ void __launch_bounds__(128) k_extend2_pack(X2Args a, int64_t ids, const ExtSegment *segs, const int64_t *slot,
                                                      const int32_t *count, const int64_t *packed_off,
                                                      ExtSegment *packed, int32_t *left, int32_t *right)
{
    const int64_t id = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (id >= ids) return;
    const int c = count[id];
    const bool none = c < 0;            // no extension on this side
    (id & 1 ? right : left)[id >> 1] = none ? 0 : a.out[id].score;
    if (none) return;
    const ExtSegment *src = segs + slot[id];
    ExtSegment *dst = packed + packed_off[id];
    if (id & 1) {
        for (int q = 0; q < c; ++q) dst[q] = src[q];
        return;
    }
    const X2Task t = x2_task(a, int(id));
    for (int q = 0; q < c; ++q) {
        const ExtSegment x = src[c - 1 - q];
        const uint32_t eh = x.h_begin + (x.type & (XT_DIAG | XT_H) ? x.length : 0);
        const uint32_t ev = x.v_begin + (x.type & (XT_DIAG | XT_V) ? x.length : 0);
        dst[q] = ExtSegment{uint32_t(t.m) - eh, uint32_t(t.n) - ev, x.length, x.type};
    }
}

__global__ void __launch_bounds__(256) k_extend2_widen(const int32_t *count, int64_t *wide, int64_t ids)
{
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i <= ids) wide[i] = i < ids && count[i] > 0 ? count[i] : 0;
}

}  // namespace gba
