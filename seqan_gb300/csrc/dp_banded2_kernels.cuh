// dp_banded2_kernels.cuh -- banded DP, two pairs of equal lengths per thread.
//
// The band phases, directions, tracked cells and extra best-cell offers are those of
// dp_banded_kernels.cuh (align/dp_algorithm_impl.h:586-967, align/dp_meta_info.h:178-370), for global
// alignments in bands of 2 to kBandFastW diagonals whose values fit 16 bits (band2_fits in
// engine.cu).  The two pairs of a thread have the same |H| and |V|, so every phase, direction and
// tracking decision is common to both and one instruction advances a cell of each: values are biased
// 16-bit halves and the trace is bit planes from sign bits, as in dp_warp2_kernels.cuh.
//
// Columns of the top, middle and bottom phases run from registers, slot k = upper - col + row (one
// per diagonal) of S and E, in one unrolled loop whose cells all take every direction; the edges are
// made by what a cell finds next to it instead of by their own code: beside the band (above slot 0,
// right of slot W - 1) lies a cell too low to win that reads as a gap extension, which leaves Upper
// and Lower cells.  In the top phase the slots above row 0 are held at the first row's start and row
// 0 at its Zero or Horizontal value; in the bottom phase the slots below row n compute what nothing
// reads.  The first and last columns take the general path from per-thread arrays.
//
// Trace: for each column, per thread five words of (D, V) masks and five of (X, Y): word k / 8 holds
// slot k in bit k % 8 of bytes 0 / 1 (D or X of the low / high pair) and 2 / 3 (V or Y).  A warp's
// column is 32 16-byte chunks of words 0-3 of (D, V), 32 of (X, Y) and, for W > 32, 32 8-byte chunks
// of the two fifth words: as many bytes a pair as the one-pair layout.
//
// Bound by issue to the ALU pipe: about 20 instructions for a cell of each pair with a trace, against
// 26 for one cell of one pair in the one-pair kernel.  1,000,000 reads of 150 bp, 33 diagonals, with
// tracebacks and CIGARs, from device memory to host buffers: 13.06 -> 6.24 ms.
#pragma once

#include "dp_banded_kernels.cuh"
#include "packed16.cuh"

#include <type_traits>

namespace gba {

constexpr int kBand2Words = (kBandFastW + 7) / 8;
// Real values lie in [kBand2Min, kBand2Max] (band2_fits).  Neighbours beside the band are below: a gap
// from them extends (E or F + ext beats S + open for gap scores from -1024 to 0), and no difference
// of two compared values reaches 2^15.
constexpr int kBand2Min = -16000, kBand2Max = 14000;
constexpr int kBand2LowE = -16200, kBand2LowS = kBand2LowE - 2 * 1024 - 64;

// Bytes of a trace column of a warp (32 threads, 64 pairs).
__host__ __device__ inline int band2_col_bytes(int W) { return W > 32 ? 1280 : 1024; }

// TraceBitMap_ byte of slot k, column col; base: the pair's trace_off, lane its lane, half 0 or 1.
__device__ __forceinline__ uint8_t trace_at_band2(const uint8_t *base, int lane, int half, int W, int upper, bool affine,
                                                  int col, int row)
{
    const int k = upper - col + row;
    if (k < 0 || k >= W) return TV_NONE;
    const uint8_t *c = base + int64_t(col) * band2_col_bytes(W);
    uint32_t dv, xy;
    if (k < 32) {
        dv = reinterpret_cast<const uint32_t *>(c)[k >> 3];
        xy = reinterpret_cast<const uint32_t *>(c + 512)[k >> 3];
    } else {
        const uint2 q = *reinterpret_cast<const uint2 *>(c + 1024 - 8 * lane);
        dv = q.x;
        xy = q.y;
    }
    const int sh = 8 * half + (k & 7);
    dv >>= sh;
    xy >>= sh;
    const uint8_t src = (dv & 1) ? TV_DIAG : ((dv >> 16) & 1 ? TV_MFV : TV_MFH);
    if (!affine) return src == TV_DIAG ? TV_DIAG : (src == TV_MFV ? uint8_t(TV_V | TV_MFV) : uint8_t(TV_H | TV_MFH));
    return uint8_t(src | ((xy & 1) ? TV_H : TV_HO) | ((xy >> 16) & 1 ? TV_V : TV_VO));
}

template <bool AFFINE, bool MATRIX, bool TRACE>
struct BandedDuo {
    static constexpr int FW = kBandFastW;
    static constexpr uint32_t ZERO2 = 0x80008000u, SET2 = 0x80008000u;   // a zero score; a "true" sign word
    const BandArgs &a;
    const int *smat;
    const uint8_t *HA, *HB, *VA, *VB;
    uint8_t *T;
    int m, n, W, lower, upper, lane;
    int INF;                          // the score of a pair none of whose cells is offered
    bool fTop, fLeft, fRight, fBottom;
    uint32_t OPEN2, EXTL, LOWS, LOWE;   // LOWS: S beside the band (linear gaps: as LOWE)
    uint32_t S[FW], E[FW], Fs[FW];
    uint32_t acc[2 * kBand2Words];    // trace words of the current column (general path)
    // caches of the current track
    uint32_t dS, vS, vF, lastF;
    // scouts (strict '>' in the reference's visiting order), one per pair
    int bs[2], be[2], bf[2], bcol[2], brow[2];

    __device__ BandedDuo(const BandArgs &args, const int *sm) : a(args), smat(sm) {}

    static __device__ __forceinline__ uint32_t both(int x) { return pack2(x + 0x8000, x + 0x8000); }
    static __device__ __forceinline__ int half(uint32_t x, int h) { return int(h ? x >> 16 : x & 0xffffu) - 0x8000; }
    static __device__ __forceinline__ uint32_t max2(uint32_t x, uint32_t y) { return __vimax3_u16x2(x, y, y); }
    static __device__ __forceinline__ uint32_t equal(uint32_t small, uint32_t large) { return small - large + 0x80008000u; }
    static __device__ __forceinline__ uint32_t signs(uint32_t x, uint32_t y) { return prmt(x, y, 0xFDB9); }

    __device__ __forceinline__ int sub1(int hc, int vc) const
    {
        if (MATRIX) return smat[((hc & 31) << 5) | (vc & 31)];
        return hc == vc ? a.match : a.mismatch;
    }
    __device__ __forceinline__ uint32_t sub(int col, int row) const
    {
        return pack2(sub1(HA[col - 1], VA[row - 1]), sub1(HB[col - 1], VB[row - 1]));
    }
    __device__ __forceinline__ void offer(uint32_t s, uint32_t e, uint32_t f, int col, int row)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (half(s, h) > bs[h]) {
                bs[h] = half(s, h);
                be[h] = half(e, h);
                bf[h] = half(f, h);
                bcol[h] = col;
                brow[h] = row;
            }
    }
    __device__ __forceinline__ int slot(int col, int row) const { return upper - col + row; }
    __device__ __forceinline__ bool in_slots(int k) const { return k >= 0 && k < W; }

    // The column's trace words to memory.
    __device__ __forceinline__ void store(int col, const uint32_t (&w)[2 * kBand2Words])
    {
        uint8_t *c = T + int64_t(col) * band2_col_bytes(W);
        *reinterpret_cast<uint4 *>(c) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4 *>(c + 512) =
            make_uint4(w[kBand2Words], w[kBand2Words + 1], w[kBand2Words + 2], w[kBand2Words + 3]);
        if (W > 32) *reinterpret_cast<uint2 *>(c + 1024 - 8 * lane) = make_uint2(w[4], w[kBand2Words + 4]);
    }

    // One cell of the general path; the horizontal neighbour (row, col - 1) is slot k + 1 of the
    // previous column, which still holds it because slots are overwritten in increasing k.
    __device__ void cell(int dir, int col, int row, bool tracked)
    {
        const int k = slot(col, row);
        const uint32_t hS = in_slots(k + 1) ? S[k + 1] : LOWS;
        const uint32_t hE = in_slots(k + 1) ? E[k + 1] : LOWE;
        uint32_t s, e = LOWE, f = vF;
        uint32_t d = 0, v = 0, x = SET2, y = SET2;     // D, V, X, Y in sign bits
        if (dir == BDIR_ZERO) {
            s = ZERO2;
            e = in_slots(k) ? E[k] : LOWE;             // stays as stored
            dS = ZERO2;
            vS = ZERO2;
        } else {
            const bool diag = dir != BDIR_HORIZONTAL && dir != BDIR_VERTICAL;
            const bool hori = dir == BDIR_ALL || dir == BDIR_HORIZONTAL || dir == BDIR_UPPER;
            const bool vert = dir == BDIR_ALL || dir == BDIR_VERTICAL || dir == BDIR_LOWER;
            const uint32_t inter = diag ? __viaddmax_u16x2(dS, sub(col, row), 0u) : 0u;
            uint32_t gh = 0, gv = 0;
            if (dir != BDIR_VERTICAL && dir != BDIR_LOWER) dS = hS;
            if (AFFINE) {
                if (hori) {
                    const uint32_t eExt = hE + EXTL;
                    e = gh = __viaddmax_u16x2(hS, OPEN2, eExt);
                    x = equal(eExt, e);
                }
                if (vert) {
                    const uint32_t fExt = vF + EXTL;
                    f = gv = __viaddmax_u16x2(vS, OPEN2, fExt);
                    y = equal(fExt, f);
                } else {
                    f = LOWE;
                }
                vF = f;
            } else {
                if (hori) gh = hS + EXTL;
                if (vert) gv = vS + EXTL;
                e = hE;
            }
            const uint32_t g = max2(gh, gv);
            s = max2(inter, g);
            d = equal(inter, s);
            v = vert ? equal(gv, g) : 0u;
            if (!diag) d = 0;
        }
        if (dir != BDIR_LOWER) vS = s;
        lastF = f;
        // Only the degenerate single-cell bands can produce a cell outside the band; it is
        // scouted but not stored.
        if (in_slots(k)) {
            S[k] = s;
            E[k] = e;
            if (TRACE) {
                acc[k >> 3] |= signs(d, v) & (0x01010101u << (k & 7));
                acc[kBand2Words + (k >> 3)] |= signs(x, y) & (0x01010101u << (k & 7));
            }
        }
        if (tracked) {
            if (in_slots(k)) Fs[k] = f;
            offer(s, e, f, col, row);
        }
    }
    __device__ __forceinline__ void begin_column()
    {
#pragma unroll
        for (int q = 0; q < 2 * kBand2Words; ++q) acc[q] = 0;
    }

    // The reference's extra best-cell offers at phase boundaries.
    __device__ void retrack(int col, int row, bool set_f)
    {
        const int k = slot(col, row);
        if (!in_slots(k)) {
            offer(ZERO2, LOWE, LOWE, col, row);
            return;
        }
        if (set_f) Fs[k] = lastF;
        offer(S[k], E[k], Fs[k], col, row);
    }

    // Register columns hIt + 1 .. of the top (slot 0 above row 0 at first), middle and bottom
    // phases.  Sr / Er: slots 0 .. W - 1, then the cell beside the band.  vw: selectors of V's codes,
    // slot k in half k & 1 of word k >> 1 (MATRIX: the codes themselves).
    enum { TOP = 0, MIDDLE = 1, BOTTOM = 2 };
    struct Regs {
        uint32_t S[FW + 1], E[FW + 1], v[FW / 2 + 1];
        uint32_t T0, T1;
        uint32_t sN, eN, fN;           // BOTTOM: the cell of row n
    };

    // Selector of row `row` (1-based) of both pairs; rows outside V read code 0.
    __device__ __forceinline__ uint32_t row_codes(int row) const
    {
        const bool in = row >= 1 && row <= n;
        const uint32_t x = in ? VA[row - 1] : 0u, y = in ? VB[row - 1] : 0u;
        return MATRIX ? ((x & 31u) | ((y & 31u) << 8)) : vsel_of((x & 7u) | ((y & 7u) << 4));
    }

    // One column.  kEdge: TOP: the slot of row 0; BOTTOM: the slot of row n.
    template <int PHASE>
    __device__ __forceinline__ void column(Regs &r, int col, int kEdge, int hA, int hB)
    {
        const uint32_t hsel = MATRIX ? 0u : ((uint32_t(hA & 7) * 0x11u) | (uint32_t(hB & 7) * 0x1100u)) * 0x00010001u;
        const int *rowA = MATRIX ? smat + ((hA & 31) << 5) : nullptr, *rowB = MATRIX ? smat + ((hB & 31) << 5) : nullptr;
        uint32_t diag = 0, up = LOWS, upF = LOWE;
        uint32_t w[2 * kBand2Words];
        if (TRACE) {
#pragma unroll
            for (int q = 0; q < 2 * kBand2Words; ++q) w[q] = 0;
        }
        const int last = W - 1;
        diag = r.S[0];
#pragma unroll
        for (int k = 0; k < FW; ++k) {
            uint32_t sb;
            if (MATRIX) {
                const uint32_t c = (k & 1) ? r.v[k >> 1] >> 16 : r.v[k >> 1];
                sb = pack2(rowA[c & 31u], rowB[(c >> 8) & 31u]);
            } else {
                const uint32_t c = r.v[k >> 1] ^ hsel;
                sb = prmt(r.T0, r.T1, (k & 1) ? c >> 16 : c);
            }
            uint32_t inter = __viaddmax_u16x2(diag, sb, 0u);
            diag = r.S[k + 1];                                   // S(row, col - 1): the next slot's diagonal
            const uint32_t hS = r.S[k + 1];
            uint32_t e = 0, f, eExt = 0, fExt = 0, g, s;
            if (PHASE == TOP && k <= kEdge) inter = fTop ? ZERO2 : 0u;   // row 0 and the slots above it
            if (AFFINE) {
                eExt = r.E[k + 1] + EXTL;
                e = __viaddmax_u16x2(hS, OPEN2, eExt);
                fExt = upF + EXTL;
                f = __viaddmax_u16x2(up, OPEN2, fExt);
            } else {
                e = hS + EXTL;
                f = up + EXTL;
            }
            if (TRACE) {
                g = max2(e, f);
                s = max2(inter, g);
                w[k >> 3] |= signs(equal(inter, s), equal(f, g)) & (0x01010101u << (k & 7));
                if (AFFINE) w[kBand2Words + (k >> 3)] |= signs(equal(eExt, e), equal(fExt, f)) & (0x01010101u << (k & 7));
            } else {
                s = __vimax3_u16x2(inter, e, f);
            }
            if (PHASE == TOP) {
                if (k <= kEdge) f = LOWE;                        // row 0 has no vertical gap
                if (k < kEdge) {                                 // above row 0: as before the first column
                    s = fTop ? ZERO2 : LOWS;
                    e = LOWE;
                }
            }
            if (PHASE == BOTTOM && k == kEdge) {
                r.sN = s;
                r.eN = e;
                r.fN = f;
            }
            r.S[k] = s;
            if (AFFINE) r.E[k] = e;
            up = s;
            upF = f;
            if (k == last) break;
        }
        if (TRACE) store(col, w);
    }

    // The next column's V window: slot k's code is the one slot k + 1 had.
    __device__ __forceinline__ void shift(Regs &r, uint32_t incoming)
    {
#pragma unroll
        for (int q = 0; q < FW / 2; ++q) r.v[q] = __funnelshift_r(r.v[q], r.v[q + 1], 16);
        r.v[FW / 2] = (r.v[FW / 2] >> 16) | (incoming << 16);
    }

    // The register phases from column hIt on (first row of the window: column hIt + 1 in slot 0);
    // leaves the state of the last column in the arrays.
    __device__ void run_fast(int &hIt, const int hTop, const int hMid, const int hBot, int &vb, int &ve)
    {
        Regs r;
        r.T0 = (uint32_t(a.match) & 0xffu) | ((uint32_t(a.mismatch) & 0xffu) * 0x01010100u);
        r.T1 = (uint32_t(a.mismatch) & 0xffu) * 0x01010101u;
        r.sN = r.eN = r.fN = LOWE;
        const uint32_t above = fTop ? ZERO2 : LOWS;
        const int virt = upper - hIt;                            // slots above row 0 in column hIt
#pragma unroll
        for (int k = 0; k <= FW; ++k) {
            r.S[k] = k < W ? (k < virt ? above : S[k < FW ? k : 0]) : LOWS;
            r.E[k] = k < W && k >= virt ? E[k < FW ? k : 0] : LOWE;
        }
        // window of column hIt + 1: slot k is row hIt + 1 - upper + k
#pragma unroll
        for (int q = 0; q <= FW / 2; ++q) {
            const int row = hIt + 1 - upper + 2 * q;
            r.v[q] = row_codes(row) | (row_codes(row + 1) << 16);
        }
        auto codes = [&]() { return row_codes(hIt + 2 - upper + FW + 1); };   // enters as column hIt + 2's last slot
        uint32_t next = codes();
        int hA = HA[hIt], hB = HB[hIt];
        auto step = [&](auto phase, int kEdge) {
            const int ca = hA, cb = hB;
            if (hIt + 1 < m) {                                   // the next column's codes, a column early
                hA = HA[hIt + 1];
                hB = HB[hIt + 1];
            }
            column<decltype(phase)::value>(r, hIt + 1, kEdge, ca, cb);
            const uint32_t in = next;
            ++hIt;
            next = codes();
            shift(r, in);
        };
        while (hIt != hTop) {
            ++ve;
            step(std::integral_constant<int, TOP>(), upper - hIt - 1);
        }
        const bool offered = fBottom && lower + n < m;           // the reference's offer after the middle phase
        while (hIt != hMid) {
            ++vb;
            ++ve;
            if (offered && hIt + 1 == hMid) step(std::integral_constant<int, BOTTOM>(), W - 1);
            else step(std::integral_constant<int, MIDDLE>(), 0);
        }
        if (offered) {
            const int k = slot(hIt, ve);                         // (no middle column: the general offer)
            if (hMid > hTop) offer(r.sN, r.eN, Fs[k], hIt, ve);
            else {
#pragma unroll
                for (int q = 0; q < FW; ++q)
                    if (q == k) offer(r.S[q], r.E[q], Fs[q], hIt, ve);
            }
        }
        while (hIt != hBot) {
            ++vb;
            const int kN = upper - hIt - 1 + n;
            step(std::integral_constant<int, BOTTOM>(), kN);
            lastF = AFFINE ? r.fN : LOWE;
            if (fBottom) {
                Fs[kN] = AFFINE ? r.fN : LOWE;
                offer(r.sN, r.eN, AFFINE ? r.fN : LOWE, hIt, n);
            }
        }
#pragma unroll
        for (int k = 0; k < FW; ++k)
            if (k < W) {
                S[k] = r.S[k];
                E[k] = AFFINE ? r.E[k] : LOWE;
            }
    }

    __device__ int first_dir(int type, int loc) const
    {
        if (type == BCOL_INITIAL) return BDIR_ZERO;
        if (loc == BLOC_FULL || loc == BLOC_TOP) return fTop ? BDIR_ZERO : BDIR_HORIZONTAL;
        return BDIR_UPPER;
    }
    __device__ int inner_dir(int type) const
    {
        if (type == BCOL_INITIAL) return fLeft ? BDIR_ZERO : BDIR_VERTICAL;
        return BDIR_ALL;
    }
    __device__ int last_dir(int type, int loc) const
    {
        if (type == BCOL_INITIAL) return fLeft ? BDIR_ZERO : BDIR_VERTICAL;
        return (loc == BLOC_TOP || loc == BLOC_MIDDLE) ? BDIR_LOWER : BDIR_ALL;
    }
    __device__ bool track_flag(int type, int loc, int which) const
    {
        const bool lastColFree = type == BCOL_FINAL && fRight;
        if (which < 2) return lastColFree;
        if (loc == BLOC_FULL || loc == BLOC_BOTTOM) return type == BCOL_FINAL || fBottom;
        return lastColFree;
    }
    __device__ void track(int col, int type, int loc, int r0, int r1)
    {
        begin_column();
        dS = LOWE; vS = LOWS; vF = LOWE;
        if (type != BCOL_INITIAL && (loc == BLOC_MIDDLE || loc == BLOC_BOTTOM) && r0 > 0 && col > 0) {
            const int kd = slot(col - 1, r0 - 1);
            dS = in_slots(kd) ? S[kd] : LOWE;
        }
        cell(first_dir(type, loc), col, r0, track_flag(type, loc, 0));
        for (int i = r0 + 1; i < r1; ++i) cell(inner_dir(type), col, i, track_flag(type, loc, 1));
        cell(last_dir(type, loc), col, r1, track_flag(type, loc, 2));
        if (TRACE) store(col, acc);
    }
    __device__ void single(int dir, int col, int row, int diag_from_col, int diag_from_row, bool tracked)
    {
        begin_column();
        dS = LOWE; vS = LOWS; vF = LOWE;
        if (diag_from_col >= 0) {
            const int kd = slot(diag_from_col, diag_from_row);
            dS = in_slots(kd) ? S[kd] : LOWE;
        }
        cell(dir, col, row, tracked);
        if (TRACE) store(col, acc);
    }

    __device__ void run()
    {
        for (int k = 0; k < W; ++k) { S[k] = LOWS; E[k] = LOWE; Fs[k] = LOWE; }
#pragma unroll
        for (int h = 0; h < 2; ++h) { bs[h] = be[h] = bf[h] = INF; bcol[h] = brow[h] = 0; }
        lastF = LOWE;
        const int lo = lower, up = upper;
        int vb = -min(0, 1 + up);
        int ve = -min(0, max(-n, lo));
        const int hb = max(0, min(m - 1, lo));
        int hTop = min(m - 1, max(0, up));
        int hMid = min(m - 1, max(0, n + lo));
        if (up > n + lo) { const int t = hTop; hTop = hMid; hMid = t; }
        const int hBot = max(0, min(m, up + n) - 1);
        if (hb == m - 1) {
            const int col = max(0, min(m, lo));
            single(BDIR_ZERO, col, 0, -1, 0, false);
            if (fRight) retrack(col, 0, false);
            return;
        }
        if (hBot == 0) {
            const int row = min(n, -up);
            single(BDIR_ZERO, 0, row, -1, 0, false);
            if (fBottom) retrack(0, row, false);
            return;
        }
        if (up < 0) {
            ++vb;
            track(0, BCOL_INITIAL, lo > -n ? BLOC_MIDDLE : BLOC_BOTTOM, vb, ve);
        } else if (lo >= 0) {
            single(BDIR_ZERO, hb, 0, -1, 0, false);
        } else {
            track(0, BCOL_INITIAL, lo <= -n ? BLOC_FULL : BLOC_TOP, vb, ve);
        }
        int hIt = hb;
        if (up >= 0 && up <= n + lo && lo > -n && hb == max(0, lo)) {
            // From the first column on, rows 0 .. col - lower (at most n) lie in slots upper - col ..
            // W - 1, then rows col - upper .. in slots 0 ..: the register phases.
            run_fast(hIt, hTop, hMid, hBot, vb, ve);
        } else {
            for (; hIt != hTop; ++hIt) {
                ++ve;
                track(hIt + 1, BCOL_INNER, BLOC_TOP, vb, ve);
            }
            if (up > n + lo) {
                if (fBottom) retrack(hIt, ve, false);
                for (; hIt != hMid; ++hIt) track(hIt + 1, BCOL_INNER, BLOC_FULL, vb, ve);
            } else {
                for (; hIt != hMid; ++hIt) {
                    ++vb; ++ve;
                    track(hIt + 1, BCOL_INNER, BLOC_MIDDLE, vb, ve);
                }
                if (fBottom && lo + n < m) retrack(hIt, ve, false);
            }
            for (; hIt != hBot; ++hIt) {
                ++vb;
                track(hIt + 1, BCOL_INNER, BLOC_BOTTOM, vb, ve);
            }
        }
        if (hIt < m - 1) {
            single(BDIR_UPPER, hIt + 1, vb + 1, hIt, vb, false);
            if (fBottom) retrack(hIt + 1, vb + 1, true);
        } else if (hIt == m - 1) {
            if (up == m - n) {
                single(BDIR_UPPER, m, vb + 1, hIt, vb, fRight);
                retrack(m, vb + 1, true);
            } else if (up >= m) {
                if (lo + n + 1 > m) {
                    ++ve;
                    track(m, BCOL_FINAL, BLOC_TOP, vb, ve);
                    if (lo + n <= m) retrack(m, ve, true);
                } else {
                    track(m, BCOL_FINAL, BLOC_FULL, vb, ve);
                }
            } else {
                ++vb;
                if (lo + n < m) {
                    track(m, BCOL_FINAL, BLOC_BOTTOM, vb, ve);
                } else {
                    ++ve;
                    track(m, BCOL_FINAL, BLOC_MIDDLE, vb, ve);
                    if (lo + n == m) retrack(m, ve, true);
                }
            }
        }
    }
};

// Slots in groups of 64: thread l of a warp runs slots l and 32 + l of its group.
template <bool AFFINE, bool MATRIX, bool TRACE>
__global__ void __launch_bounds__(128, 3) k_dp_banded2(BandArgs a)
{
    extern __shared__ int smat[];
    if (MATRIX) {
        for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
            const int r = i >> 5, c = i & 31;
            smat[i] = (r < a.alphabet && c < a.alphabet) ? a.matrix[r * a.alphabet + c] : 0;
        }
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int64_t group = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t slot = group * 64 + lane;
    if (slot >= a.num_slots) return;
    const int pA = a.order[slot], pB = a.order[slot + 32];
    if (pA < 0) return;
    const PairDesc A = a.pairs[pA], B = a.pairs[pB];
    BandedDuo<AFFINE, MATRIX, TRACE> bp(a, smat);
    bp.lane = lane;
    bp.m = A.m;
    bp.n = A.n;
    bp.INF = A.inf;
    bp.W = a.upper - a.lower + 1;
    bp.lower = a.lower;
    bp.upper = a.upper;
    bp.HA = a.seq_h + A.h_off;
    bp.HB = a.seq_h + B.h_off;
    bp.VA = a.seq_v + A.v_off;
    bp.VB = a.seq_v + B.v_off;
    bp.T = TRACE ? a.trace + A.trace_off : nullptr;
    bp.fTop = a.free_ends & FREE_TOP;
    bp.fLeft = a.free_ends & FREE_LEFT;
    bp.fRight = a.free_ends & FREE_RIGHT;
    bp.fBottom = a.free_ends & FREE_BOTTOM;
    bp.OPEN2 = AFFINE ? pack2(a.gap_open, a.gap_open) : pack2(a.gap_extend, a.gap_extend);
    bp.EXTL = uint32_t(a.gap_extend) * 0x00010001u;
    bp.LOWS = bp.both(AFFINE ? kBand2LowS : kBand2LowE);
    bp.LOWE = bp.both(kBand2LowE);
    bp.run();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = h ? pB : pA;
        a.score[p] = bp.bs[h];
        if (a.end_h) a.end_h[p] = bp.bcol[h];
        if (a.end_v) a.end_v[p] = bp.brow[h];
        if (a.best_e) a.best_e[p] = bp.be[h];
        if (a.best_f) a.best_f[p] = bp.bf[h];
    }
}

}  // namespace gba
