// dp_warp2_kernels.cuh -- packed 16-bit warp bands: 64 strips per warp, two cells per instruction.
//
// For pairs whose every cell value fits 16 bits (w2_fits in engine.cu), one warp computes a band of
// 64 strips of R rows of one pair.  Lane l owns strip l in the low 16-bit halves of its registers
// and strip 32 + l in the high halves, so every max / add-max instruction advances two cells.  The
// strips form an anti-diagonal front: at step t the low half of lane l is at column t - l and the
// high half at column t - l - 32; each step lane l receives the bottom row (S, F) of lane l - 1 by
// one rotating shuffle, and lane 0's high half receives lane 31's low half (strip 31 is the strip
// above strip 32).  A band takes m + 64 steps.
//
// Rows per strip.  R is chosen per pair by the planner (PairDesc::rows; w2_rows and the task list in
// engine.cu).  A step has a fixed part (hand-off, loop), so a pair takes as few bands as possible and
// the smallest R that covers its rows in them (a band was 256 rows whatever the pair held: a 300-row
// protein paid for 384 rows in two bands, now for 320 in one).  A pair that would keep one warp busy
// while most of the device has nothing left to do is cut into more bands of fewer rows, which run
// as separate tasks on different warps at the same time.
//
// Bound by issue to the ALU pipe in full batches (85% busy in the protein search), and by the
// latency of a lone warp's own instructions where one pair or few are in flight.  Measured, whole
// calls, before and after this form of the kernel (rows per pair, score profile, biased values, self-
// validating row entries, no size limits): protein search (350 residues against 20,000) 3.11 ->
// 1.77 ms; 20,000 protein pairs with tracebacks 5.02 -> 3.95 ms; 2,000 pairs of 100 to 10,000 bp with
// tracebacks (32-bit kernel before) 8.9 -> 5.2 ms; 8 pairs of 10,000 bp (likewise) 5.09 -> 2.58 ms.
//
// Bands of one pair hand their bottom row (strip 63: lane 31, high half) on through global memory,
// one 64-bit entry per column: the packed (S, F) and a tag naming the band that wrote it.  An entry
// is written and read whole, so the reader polls the data itself and needs no flag or fence; it
// reads kW2Chunk columns ahead.  Band b writes slot b & 1 of two and reads slot (b - 1) & 1: band
// b + 2 writes column j only after band b + 1 produced it, which it did after reading column j of
// band b.  Every band waited on was taken from the queue earlier by a running warp, and each wait
// has an iteration limit after which the kernel records an error and carries on.  Pairs whose bands
// run in order on one warp use one slot, rewritten in place, and no waits.
//
// Values are kept with a bias of 0x8000, so that every real value is a non-negative 16-bit number:
// the maxima are the unsigned DPX ones, and adding the same constant to both halves, or taking the
// difference of two ordered values, is one 32-bit integer add, exact in both halves.
//
// Recurrences, tie rules and tracked cells are the reference's (align/dp_formula_affine.h:66-330,
// align/dp_formula_linear.h:62-258, align/dp_meta_info.h:178-221, align/dp_scout.h:166-180), in
// the max / add-max form whose values equal the compare-and-select ones, ties included:
//   E = max(E_left + ext, S_left + open)   (extend wins ties)
//   F = max(F_up + ext, S_up + open)       (extend wins ties)
//   G = max(E, F), S = max(diag + sub, G)  (F wins ties against E, the diagonal against G)
// and for linear gaps G = max(S_left + g, S_up + g) (vertical wins ties).  Local mode floors S at 0.
//
// Trace: what _doTraceback (align/dp_traceback_impl.h:376-450) reads of the TraceBitMap_ byte
// (align/dp_profile.h:121-135), one bit plane per question:
//   D: S == diag + sub     V: G == F     X: E == E_left + ext     Y: F == F_up + ext
//   and in local mode Z: S == 0
// The source of S is none with Z, else the diagonal with D, else vertical with V, else horizontal.
// The oracle checks (tests/test_trace4_oracle.py) that this much gives the reference's traceback on
// every configuration.  A question's answer for both halves is the sign bits of 0x8000 - (larger -
// smaller), one three-input add; one byte permute turns the signs of two questions into byte masks
// and one logic operation puts them into the lane's trace word (w2_trace_at has the bit places).
// Row 0 is stored as TraceBitMap_ bytes, as in the other layouts.
#pragma once

#include "dp_common.cuh"
#include "dp_warp_kernels.cuh"
#include "packed16.cuh"

namespace gba {

constexpr int kW2Chunk = 8;                    // columns a band reads ahead of its front
constexpr int kW2Inf = -31680;                 // "infinity": below every real value, and still a
                                               // non-negative biased number after one gap score (<= 1024)
constexpr int kW2Bias = 0x8000;

// How a column's substitution scores are looked up.
enum { W2_EQUAL = 0, W2_PROFILE = 1, W2_TABLE = 2 };
// Rows per strip: at most 8; 6 where the trace has five planes; 4 with the table lookup, which
// keeps two registers per row.
__host__ __device__ inline int w2_max_rows(int mat, bool local, bool trace)
{
    return mat == W2_TABLE ? 4 : (local && trace ? 6 : 8);
}

// Trace bytes of one lane and step.
__host__ __device__ inline int w2_trace_word(int R, bool local)
{
    return R == 2 && !local ? 2 : (R <= (local ? 3 : 4) ? 4 : 8);
}

__host__ __device__ inline int w2_bands(int n, int R) { return (n + 64 * R - 1) / (64 * R); }

__host__ __device__ inline int64_t w2_band_off(int m, int b, int R, bool local)
{
    return align16(m + 1) + int64_t(b) * (m + 64) * 32 * w2_trace_word(R, local);
}

// Trace bytes of one pair: row 0 (m + 1 bytes, padded), then per band m + 64 steps of 32 lanes.
__host__ __device__ inline int64_t w2_trace_bytes(int m, int n, int R, bool local)
{
    return w2_band_off(m, n > 0 ? w2_bands(n, R) : 0, R, local);
}

// Byte offset of the trace word that holds cell (col, row) within the pair's trace (row 0: the
// cell's byte).
__device__ __forceinline__ int64_t w2_trace_off(int m, int R, bool local, int col, int row)
{
    if (row == 0) return col;
    const int s = (row - 1) / R;
    return w2_band_off(m, s >> 6, R, local) + (int64_t(col + (s & 63)) * 32 + (s & 31)) * w2_trace_word(R, local);
}

// TraceBitMap_ byte of cell (col, row).  Bytes 0 / 1 of the words are the low / high strip's D (and
// X), bytes 2 / 3 its V (and Y); row r of the strip is bit r.  X and Y lie four bits up in the same
// word for R <= 4, else in a second word.  Z goes by row pairs, even rows in bytes 0 / 1, odd ones
// in bytes 2 / 3, in bits that the others leave free.
__host__ __device__ inline int w2_zero_bit(int R, int q)   // bit of row pair q; + 32: the second word
{
    return R == 2 ? 2 : R == 3 ? 3 + 4 * q : R == 4 ? 32 + q : q < 2 ? 6 + q : 32 + 6;
}
__device__ __forceinline__ uint8_t w2_trace_at(const uint8_t *base, int m, int R, bool local, bool affine, int col,
                                               int row)
{
    const uint8_t *w = base + w2_trace_off(m, R, local, col, row);
    if (row == 0) return *w;
    const int s = (row - 1) / R, r = row - 1 - s * R, h = (s >> 5) & 1;
    uint32_t w0, w1 = 0;
    if (w2_trace_word(R, local) == 2) {
        // bits 2, 3, 6, 7 of each byte hold what the other words have in bytes 2 and 3
        w0 = *reinterpret_cast<const uint16_t *>(w);
        w0 |= (w0 & 0xccccu) << 14;
    } else if (w2_trace_word(R, local) == 8) {
        const uint2 q = *reinterpret_cast<const uint2 *>(w);
        w0 = q.x;
        w1 = q.y;
    } else {
        w0 = *reinterpret_cast<const uint32_t *>(w);
    }
    if (local) {
        const int zb = w2_zero_bit(R, r >> 1);
        if (((zb >= 32 ? w1 : w0) >> ((zb & 31) + 8 * (h + 2 * (r & 1)))) & 1) return TV_NONE;
    }
    const int sh = 8 * h + r;
    const int src = (w0 >> sh) & 1 ? TV_DIAG : ((w0 >> (sh + 16)) & 1 ? TV_MFV : TV_MFH);
    if (!affine) return src == TV_DIAG ? TV_DIAG : (src == TV_MFV ? (TV_V | TV_MFV) : (TV_H | TV_MFH));
    const uint32_t gaps = R <= 4 ? w0 >> (sh + 4) : w1 >> sh;
    return uint8_t(src | (gaps & 1 ? TV_H : TV_HO) | ((gaps >> 16) & 1 ? TV_V : TV_VO));
}

struct Warp2Args {
    const uint8_t *seq_h;
    const uint8_t *seq_v;
    const PairDesc *pairs;
    const int2 *tasks;             // (pair, band): band -1 = all bands of the pair in order on one warp
    uint64_t *rowbuf;              // per multi-band pair at rowbuf_off[p]: 1 (in order) or 2 (pipelined;
                                   // zeroed per run) slots of m + 1 entries
    const int64_t *rowbuf_off;
    BandState *bands;              // pipelined pairs at band_base[p]: one per band (zeroed per run)
    const int64_t *band_base;
    int32_t *error;                // set to 1 when a wait between bands ran out
    uint8_t *trace;
    int32_t *score, *end_h, *end_v, *best_e, *best_f;
    const int32_t *matrix;
    int32_t *task_counter;
    int32_t num_tasks;
    int32_t match, mismatch, gap_open, gap_extend;
    int32_t free_ends;
    int32_t alphabet;
};

// Shared memory of a block with profiles: per warp `alphabet` letters x 2 halves x 32 lanes x 8 rows,
// then a letter of zeros for codes outside the alphabet.  27 letters let four blocks share an SM.
constexpr int kW2Warps = 4;
__host__ __device__ inline size_t w2_profile_bytes(int alphabet) { return size_t(alphabet) * 512; }
__host__ __device__ inline size_t w2_shared_bytes(int mat, int alphabet)
{
    return mat == W2_PROFILE ? kW2Warps * w2_profile_bytes(alphabet) + 512 : 0;
}

// Best cell of one half-strip (column-major first maximum).
struct Best1 {
    int s, e, f, col, row;
    __device__ __forceinline__ void offer(int cs, int ce, int cf, int ccol, int crow)
    {
        if (cs >= s && (cs > s || ccol < col || (ccol == col && crow < row))) {
            s = cs; e = ce; f = cf; col = ccol; row = crow;
        }
    }
    // For candidates that arrive in column-major order: a later cell wins only with a higher score.
    __device__ __forceinline__ void offer_later(int cs, int ce, int cf, int ccol, int crow)
    {
        if (cs > s) { s = cs; e = ce; f = cf; col = ccol; row = crow; }
    }
};

__device__ __forceinline__ uint32_t w2_sel(uint32_t x, uint32_t mask, uint32_t y)
{
    return (x & ~mask) | (y & mask);   // one LOP3
}
__device__ __forceinline__ uint32_t w2_max(uint32_t a, uint32_t b) { return __vimax3_u16x2(a, b, b); }

// Biased halves and back.
__device__ __forceinline__ uint32_t w2_pack(int lo, int hi) { return pack2(lo + kW2Bias, hi + kW2Bias); }
__device__ __forceinline__ int w2_lo(uint32_t x) { return int(x & 0xffffu) - kW2Bias; }
__device__ __forceinline__ int w2_hi(uint32_t x) { return int(x >> 16) - kW2Bias; }

// Both halves: the sign bit is set where `small` (<= `large`) equals it.
__device__ __forceinline__ uint32_t w2_equal(uint32_t small, uint32_t large) { return small - large + 0x80008000u; }
// The sign bits of a's and b's halves as byte masks: a low, a high, b low, b high.
__device__ __forceinline__ uint32_t w2_signs(uint32_t a, uint32_t b) { return prmt(a, b, 0xFDB9); }

// S(0, j) of row 0 (Horizontal gaps, or Zero with a free first row); E(0, j) equals it for j >= 1.
__device__ __forceinline__ int w2_row0(int j, bool fTop, bool affine, int open, int ext)
{
    if (fTop || j == 0) return 0;
    return affine ? open + (j - 1) * max(ext, open) : j * ext;
}

__device__ __forceinline__ uint64_t w2_ld_entry(const uint64_t *p)
{
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void w2_st_entry(uint64_t *p, uint64_t v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Per-lane state of one band: lane l holds strip l (low halves) and strip 32 + l (high halves).
template <bool AFFINE, bool LOCAL, int MAT, bool TRACE, int R>
struct W2Lane {
    uint32_t vsel[R];              // W2_EQUAL: PRMT selectors of the two halves' row codes
    int vlo[R], vhi[R];            // W2_TABLE: row codes of the low / high strip
    const uint8_t *prof;           // W2_PROFILE: this lane's 8 score bytes of letter 0, low strip
    uint32_t selS, selF, selH;     // hand-off selectors (lane 0 takes the band's inputs)
    int nlo, nhi;                  // rows of the two strips inside the matrix
    int i0lo, i0hi;                // first rows of the two strips
    int rowNlo, rowNhi;            // index of row n in each strip, or -1
    uint32_t Sp[R], Ep[R], Fp[R];
    uint32_t diagNext, outS, outF, hcode;
    uint32_t bestS2;               // bl.s and bh.s packed (LOCAL)
    Best1 bl, bh;

    __device__ __forceinline__ uint32_t rowmask(int r) const
    {
        return (r < nlo ? 0x0000ffffu : 0u) | (r < nhi ? 0xffff0000u : 0u);
    }

    // x[i] by selection: an index that is not a constant would move the arrays to local memory.
    static __device__ __forceinline__ uint32_t pick(const uint32_t (&x)[R], int i)
    {
        uint32_t v = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) v |= x[r] & (r == i ? 0xffffffffu : 0u);
        return v;
    }

    // One step t; above / hnew: the band's input in column t, (S, F) of the row above and the code of
    // H.  EDGE: some half may be at column 0 or outside [1, m - 1] (fill and drain).
    template <bool EDGE>
    __device__ __forceinline__ void step(const int *smat, int t, int lane, int m, int n, uint32_t above, uint32_t hnew,
                                         uint8_t *tstore, uint32_t T0, uint32_t T1, uint32_t OPEN2, uint32_t EXTL,
                                         bool fLeft, bool fRight, bool fBottom)
    {
        const uint32_t ZERO2 = 0x80008000u, INF2 = w2_pack(kW2Inf, kW2Inf);
        // Hand-off: lane l takes lane l - 1's bottom row; lane 0 takes the row above the band (low
        // half) and lane 31's low half (high half).  Column codes rotate the same way.
        const int from = (lane + 31) & 31;
        const uint32_t rotS = __shfl_sync(0xffffffffu, outS, from);
        const uint32_t rotF = AFFINE ? __shfl_sync(0xffffffffu, outF, from) : 0u;
        const uint32_t rotH = __shfl_sync(0xffffffffu, hcode, from);
        uint32_t sUp = prmt(above, rotS, selS);
        uint32_t fUp = AFFINE ? prmt(above, rotF, selF) : 0u;
        const uint32_t hcur = hcode;
        hcode = prmt(hnew, rotH, selH);
        const int jlo = t - lane, jhi = jlo - 32;
        uint32_t m0 = 0;                // halves at column 0
        if (EDGE) m0 = (jlo == 0 ? 0x0000ffffu : 0u) | (jhi == 0 ? 0xffff0000u : 0u);
        uint32_t diag = diagNext;
        diagNext = sUp;
        uint32_t plo[2], phi[2];
        if (MAT == W2_PROFILE) {
            const uint8_t *ql = prof + (hcur & 0xffffu), *qh = prof + (hcur >> 16) + 256;
            if (R > 4) {
                const uint2 x = *reinterpret_cast<const uint2 *>(ql), y = *reinterpret_cast<const uint2 *>(qh);
                plo[0] = x.x; plo[1] = x.y;
                phi[0] = y.x; phi[1] = y.y;
            } else {
                plo[0] = plo[1] = *reinterpret_cast<const uint32_t *>(ql);
                phi[0] = phi[1] = *reinterpret_cast<const uint32_t *>(qh);
            }
        }
        const int hrlo = int(hcur & 0xffffu), hrhi = int(hcur >> 16);
        uint32_t acc0 = 0, acc1 = 0, zprev = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            uint32_t sub;
            if (MAT == W2_PROFILE)
                sub = prmt(plo[r >> 2], phi[r >> 2], uint32_t(0xC480 + 0x1111 * (r & 3)));
            else if (MAT == W2_TABLE)
                sub = prmt(uint32_t(smat[hrlo + vlo[r]]), uint32_t(smat[hrhi + vhi[r]]), 0x5410);
            else
                sub = prmt(T0, T1, hcur ^ vsel[r]);
            uint32_t inter = __viaddmax_u16x2(diag, sub, 0u);
            if (EDGE) inter &= ~m0;
            diag = Sp[r];
            uint32_t s, g = 0, e = 0, f, eExt = 0, fExt = 0;
            if (AFFINE) {
                eExt = Ep[r] + EXTL;
                e = __viaddmax_u16x2(Sp[r], OPEN2, eExt);
                if (EDGE) {
                    eExt = w2_sel(eExt, m0, INF2);
                    e = w2_sel(e, m0, INF2);
                }
                fExt = fUp + EXTL;
                f = __viaddmax_u16x2(sUp, OPEN2, fExt);
                if (TRACE) g = w2_max(e, f);
            } else {
                f = sUp + EXTL;
                e = Sp[r] + EXTL;
                if (EDGE) e &= ~m0;                        // column 0: vertical only
                if (TRACE) g = w2_max(e, f);
            }
            if (TRACE) {
                s = LOCAL ? __vimax3_u16x2(inter, g, ZERO2) : w2_max(inter, g);
            } else {
                s = __vimax3_u16x2(inter, e, f);
                if (LOCAL) s = w2_max(s, ZERO2);
            }
            if (EDGE && (LOCAL || fLeft)) {
                s = w2_sel(s, m0, ZERO2);                  // Zero cells of a free first column
                if (AFFINE) f = w2_sel(f, m0, fUp);        // F passes through unchanged
            }
            if (TRACE) {
                acc0 |= w2_signs(w2_equal(inter, s), w2_equal(f, g)) & (0x01010101u << r);
                if (AFFINE) {
                    const uint32_t x = w2_signs(w2_equal(eExt, e), w2_equal(fExt, f));
                    if (R <= 4) acc0 |= x & (0x10101010u << r);
                    else acc1 |= x & (0x01010101u << r);
                }
                if (LOCAL) {
                    const uint32_t z = w2_equal(ZERO2, s);
                    if ((r & 1) || r == R - 1) {
                        const uint32_t x = (r & 1) ? w2_signs(zprev, z) : w2_signs(z, 0u);
                        constexpr int kWord = 32;
                        const int zb = w2_zero_bit(R, r >> 1);
                        if (zb >= kWord) acc1 |= x & (0x01010101u << (zb & 31));
                        else acc0 |= x & (0x01010101u << (zb & 31));
                    }
                    zprev = z;
                }
            }
            Sp[r] = s;
            if (AFFINE) Ep[r] = e;
            Fp[r] = f;
            sUp = s;
            fUp = f;
        }
        if (TRACE) {
            if (w2_trace_word(R, LOCAL) == 8) *reinterpret_cast<uint2 *>(tstore) = make_uint2(acc0, acc1);
            else if (w2_trace_word(R, LOCAL) == 4) *reinterpret_cast<uint32_t *>(tstore) = acc0;
            else *reinterpret_cast<uint16_t *>(tstore) = uint16_t(acc0 | (acc0 >> 14));
        }
        outS = sUp;
        outF = fUp;

        // Tracked cells.
        if (LOCAL) {
            // Rows beyond n: with a profile their substitution scores are -128, so they never exceed
            // the real cell they come from; otherwise they are masked.
            uint32_t mx;
            if (MAT != W2_PROFILE && nhi < R) {
                mx = Sp[0] & rowmask(0);
#pragma unroll
                for (int r = 1; r < R; ++r) mx = w2_max(mx, Sp[r] & rowmask(r));
            } else {
                mx = Sp[0];
#pragma unroll
                for (int r = 1; r + 1 < R; r += 2) mx = __vimax3_u16x2(mx, Sp[r], Sp[r + 1]);
                if (!(R & 1)) mx = w2_max(mx, Sp[R - 1]);
            }
            if (EDGE)
                mx &= (jlo >= 1 && jlo <= m ? 0x0000ffffu : 0u) | (jhi >= 1 && jhi <= m ? 0xffff0000u : 0u);
            if (w2_max(mx, bestS2) != bestS2) {
                // The first row holding each half's maximum, with its E and F, found for both halves
                // at once (bottom up, so the first matching row is the last one selected).
                uint32_t ridx = 0, es = 0, fs = 0;
#pragma unroll
                for (int r = R - 1; r >= 0; --r) {
                    uint32_t eq = __vcmpeq2(Sp[r], mx);
                    if (MAT != W2_PROFILE) eq &= rowmask(r);
                    ridx = w2_sel(ridx, eq, uint32_t(r) * 0x00010001u);
                    if (TRACE) {
                        es = w2_sel(es, eq, Ep[r]);
                        fs = w2_sel(fs, eq, Fp[r]);
                    }
                }
                const int mlo = w2_lo(mx), mhi = w2_hi(mx);
                if (mlo > bl.s) bl.offer_later(mlo, w2_lo(es), w2_lo(fs), jlo, i0lo + int(ridx & 0xffffu));
                if (mhi > bh.s) bh.offer_later(mhi, w2_hi(es), w2_hi(fs), jhi, i0hi + int(ridx >> 16));
                bestS2 = w2_pack(max(bl.s, kW2Inf), max(bh.s, kW2Inf));
            }
        } else {
            // Global: the last column (every row with a free last column, else row n) and, with a
            // free last row, row n of every column (column 0 included).
            const bool lastLo = EDGE && jlo == m, lastHi = EDGE && jhi == m;
            if (EDGE && fRight) {
                // A lane meets one last column per half: every row, r a constant.
                if (lastLo) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (r < nlo) bl.offer_later(w2_lo(Sp[r]), jlo == 0 ? -(1 << 30) : w2_lo(Ep[r]), w2_lo(Fp[r]), jlo, i0lo + r);
                }
                if (lastHi) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (r < nhi) bh.offer_later(w2_hi(Sp[r]), jhi == 0 ? -(1 << 30) : w2_hi(Ep[r]), w2_hi(Fp[r]), jhi, i0hi + r);
                }
            }
            if (rowNlo >= 0 && (lastLo || (fBottom && jlo >= 0 && jlo <= m)))
                bl.offer_later(w2_lo(pick(Sp, rowNlo)), jlo == 0 ? -(1 << 30) : w2_lo(pick(Ep, rowNlo)),
                               w2_lo(pick(Fp, rowNlo)), jlo, n);
            if (rowNhi >= 0 && (lastHi || (fBottom && jhi >= 0 && jhi <= m)))
                bh.offer_later(w2_hi(pick(Sp, rowNhi)), jhi == 0 ? -(1 << 30) : w2_hi(pick(Ep, rowNhi)),
                               w2_hi(pick(Fp, rowNhi)), jhi, n);
        }
    }
};

// The band's inputs, kW2Chunk columns at a time in lanes 0 .. kW2Chunk - 1: the row above ((S, F)
// packed) and the codes of H in the form the lookup takes, loaded one chunk ahead.
template <int MAT>
struct W2Input {
    const uint8_t *H;
    const uint64_t *row;           // band b - 1's entries, or null for band 0
    uint32_t tag;                  // that its entries carry; 0: no check (bands in order)
    int m, lane;
    bool fTop, affine;
    int open, ext;
    int alphabet;
    uint32_t outside;              // W2_PROFILE: offset of the letter of zeros
    uint32_t above, code;          // the current chunk
    uint64_t next;                 // of the next chunk: the loaded entry and code
    int nextCode;

    __device__ __forceinline__ void load_row(int c0)
    {
        if (row && lane < kW2Chunk && c0 + lane <= m) next = w2_ld_entry(row + c0 + lane);
    }
    __device__ __forceinline__ void load(int c0)
    {
        load_row(c0);
        nextCode = H[min(c0 + (lane & (kW2Chunk - 1)), m - 1)];
    }
    // Makes the chunk at c0 (loaded before) the current one, waiting until its entries are there,
    // and loads the next.  Lanes past column m keep the row above that they have: a strip's low half runs
    // 32 columns ahead of its high one, so it is past m while the high half holds real cells, and beside
    // a value from elsewhere (a zero, say) a cell with a score near the range's ends could differ from
    // its neighbours by more than 2^15, which w2_equal would carry into the high half.
    __device__ __forceinline__ void advance(int c0, int32_t *error)
    {
        const int c = c0 + (lane & (kW2Chunk - 1));
        if (row) {
            const bool mine = lane < kW2Chunk && c <= m;
            if (tag) {
                for (int it = 0; !__all_sync(0xffffffffu, !mine || uint32_t(next >> 32) == tag); ++it) {
                    // Gives up after about a second, or when another wait already gave up.
                    if ((it & 255) == 255 && __any_sync(0xffffffffu, *(volatile int32_t *)error != 0)) break;
                    if (it > (1 << 20)) {
                        if (lane == 0) atomicExch(error, 1);
                        break;
                    }
                    if (it > 32) __nanosleep(64);
                    load_row(c0);
                }
            }
            if (c <= m) above = uint32_t(next);
            if (c0 == 0 && m < kW2Chunk - 1) above = __shfl_sync(0xffffffffu, uint32_t(next), min(lane, m));
        } else {
            above = w2_pack(w2_row0(c, fTop, affine, open, ext), kW2Inf);
        }
        const int x = nextCode;
        code = MAT == W2_EQUAL ? uint32_t((x & 7) * 0x11u)
               : MAT == W2_TABLE ? uint32_t((x & 31) << 5)
               : (x & 31) < alphabet ? uint32_t((x & 31) << 9) : outside;
        load(c0 + kW2Chunk);
    }
};

// Band b of pair p (all lanes).  R: rows per half-strip.  seq: the pair's bands run in order on this
// warp (best cell carried in `carry`); else this band is a pipelined task.
template <bool AFFINE, bool LOCAL, int MAT, bool TRACE, int R>
__device__ __forceinline__ void warp2_band(const Warp2Args &a, const int *smat, const int8_t *bmat, uint8_t *profile,
                                           uint32_t outside, int p, int b, int lane, bool seq, Best1 &carry)
{
    const PairDesc d = a.pairs[p];
    const int m = d.m, n = d.n;
    const int bands = w2_bands(n, R);
    const uint8_t *H = a.seq_h + d.h_off;
    const uint8_t *V = a.seq_v + d.v_off;
    uint8_t *T = TRACE ? a.trace + d.trace_off : nullptr;
    const int fe = LOCAL ? (FREE_TOP | FREE_LEFT | FREE_RIGHT | FREE_BOTTOM) : a.free_ends;
    const bool fTop = fe & FREE_TOP, fLeft = fe & FREE_LEFT;
    const bool fRight = fe & FREE_RIGHT, fBottom = fe & FREE_BOTTOM;
    const int OPEN = AFFINE ? a.gap_open : a.gap_extend;
    const int EXT = a.gap_extend;
    const uint32_t OPEN2 = pack2(OPEN, OPEN);
    const uint32_t EXTL = uint32_t(EXT) * 0x00010001u;     // adds EXT to both halves
    const uint32_t T0 = (uint32_t(a.match) & 0xffu) | ((uint32_t(a.mismatch) & 0xffu) * 0x01010100u);
    const uint32_t T1 = (uint32_t(a.mismatch) & 0xffu) * 0x01010101u;
    const int NONE = -(1 << 30);
    const uint32_t INF2 = w2_pack(kW2Inf, kW2Inf);

    W2Lane<AFFINE, LOCAL, MAT, TRACE, R> w;
    const int rowBase = b * 64 * R;
    w.i0lo = rowBase + lane * R + 1;
    w.i0hi = rowBase + (32 + lane) * R + 1;
    w.nlo = min(max(n - w.i0lo + 1, 0), R);
    w.nhi = min(max(n - w.i0hi + 1, 0), R);
    w.rowNlo = (n >= w.i0lo && n < w.i0lo + R) ? n - w.i0lo : -1;
    w.rowNhi = (n >= w.i0hi && n < w.i0hi + R) ? n - w.i0hi : -1;
    if (MAT == W2_PROFILE) w.prof = profile + lane * 8;
    w.selS = lane ? 0x7654u : 0x5410u;
    w.selF = lane ? 0x7654u : 0x5432u;
    w.selH = lane ? 0x7654u : (MAT == W2_EQUAL ? 0x1140u : 0x5410u);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int clo = r < w.nlo ? V[w.i0lo + r - 1] : 0;
        const int chi = r < w.nhi ? V[w.i0hi + r - 1] : 0;
        if (MAT == W2_EQUAL) {
            w.vsel[r] = vsel_of(uint32_t(clo & 7) | (uint32_t(chi & 7) << 4));
        } else {
            w.vlo[r] = clo & 31;
            w.vhi[r] = chi & 31;
        }
        w.Sp[r] = INF2;
        w.Ep[r] = INF2;
        w.Fp[r] = INF2;
    }
    if (MAT == W2_PROFILE) {
        // The score bytes of this lane's rows against every letter of H: one 8-byte (4-byte) read
        // per half and step gives the scores of all rows.
        __syncwarp();
        for (int c = 0; c < a.alphabet; ++c) {
            uint32_t lo[2] = {0, 0}, hi[2] = {0, 0};
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint32_t x = r < w.nlo ? uint8_t(bmat[c * 32 + w.vlo[r]]) : 0x80u;
                const uint32_t y = r < w.nhi ? uint8_t(bmat[c * 32 + w.vhi[r]]) : 0x80u;
                lo[r >> 2] |= x << (8 * (r & 3));
                hi[r >> 2] |= y << (8 * (r & 3));
            }
            *reinterpret_cast<uint2 *>(profile + c * 512 + lane * 8) = make_uint2(lo[0], lo[1]);
            *reinterpret_cast<uint2 *>(profile + c * 512 + 256 + lane * 8) = make_uint2(hi[0], hi[1]);
        }
        __syncwarp();
    }
    w.diagNext = INF2;
    w.outS = INF2;
    w.outF = INF2;
    w.hcode = 0;
    w.bl = Best1{NONE, NONE, NONE, 0, 0};
    w.bh = Best1{NONE, NONE, NONE, 0, 0};
    Best1 row0{NONE, NONE, NONE, 0, 0};    // candidates of row 0 (not in column-major order here)
    if (b == 0) {
        if (LOCAL && lane == 0) row0.offer(0, NONE, NONE, 0, 0);
        if (!LOCAL && fRight && lane == 0)
            row0.offer(w2_row0(m, fTop, AFFINE, OPEN, EXT), fTop ? NONE : w2_row0(m, fTop, AFFINE, OPEN, EXT), NONE, m, 0);
        if (TRACE) {
            // Row 0: Zero at (0, 0) and with a free first row, else Horizontal (open at column 1).
            for (int c = lane; c <= m; c += 32) {
                uint8_t tv = TV_NONE;
                if (c >= 1 && !fTop)
                    tv = AFFINE ? ((c == 1 || EXT < OPEN) ? (TV_HO | TV_MFH) : (TV_H | TV_MFH)) : (TV_H | TV_MFH);
                T[c] = tv;
            }
        }
    }
    // Local scores start from 0: a cell of score 0 never beats the best cell (0, 0).
    w.bestS2 = LOCAL ? 0x80008000u : INF2;
    if (LOCAL) w.bl.s = w.bh.s = 0, w.bl.col = w.bh.col = INT_MAX;

    uint64_t *rowOut = nullptr;
    W2Input<MAT> in{};
    BandState *st = nullptr;
    if (bands > 1) {
        uint64_t *base = a.rowbuf + a.rowbuf_off[p];
        rowOut = seq ? base : base + int64_t(b & 1) * (m + 1);
        if (b > 0) in.row = seq ? base : base + int64_t((b + 1) & 1) * (m + 1);
        if (!seq) st = a.bands + a.band_base[p] + b;
    }
    in.H = H;
    in.tag = seq ? 0 : uint32_t(b);         // band b - 1 tags its entries with b
    in.m = m;
    in.lane = lane;
    in.fTop = fTop;
    in.affine = AFFINE;
    in.open = OPEN;
    in.ext = EXT;
    in.alphabet = a.alphabet;
    in.outside = outside;
    in.load(0);
    constexpr int kWord = TRACE ? 32 * (R == 2 && !LOCAL ? 2 : (R <= (LOCAL ? 3 : 4) ? 4 : 8)) : 0;
    uint8_t *Tb = TRACE ? T + w2_band_off(m, b, R, LOCAL) + lane * (kWord / 32) : nullptr;
    uint64_t *out = b + 1 < bands && lane == 31 ? rowOut - 63 : nullptr;   // column t - 63 at step t
    const uint64_t tag = uint64_t(uint32_t(b + 1)) << 32;
    const int last = m + 63;

    // Steps 64 .. m - 1 have every half in columns 1 .. m - 1 (no column 0, no last column);
    // the fill and drain steps around them take the edge path.
#define GBA_W2_STEP(EDGE)                                                                                  \
    do {                                                                                                   \
        if ((t & (kW2Chunk - 1)) == 0) in.advance(t, a.error);                                             \
        const uint32_t above = __shfl_sync(0xffffffffu, in.above, t & (kW2Chunk - 1));                     \
        const uint32_t code = __shfl_sync(0xffffffffu, in.code, t & (kW2Chunk - 1));                       \
        w.template step<EDGE>(smat, t, lane, m, n, above, code, Tb, T0, T1, OPEN2, EXTL, fLeft, fRight, fBottom); \
        Tb += kWord;                                                                                       \
        if (out && (!(EDGE) || (t >= 63 && t <= m + 63))) w2_st_entry(out + t, tag | prmt(w.outS, w.outF, 0x7632)); \
        ++t;                                                                                               \
    } while (0)
    int t = 0;
    while (t <= last) {
        if (t >= 64 && t < m) {
            do GBA_W2_STEP(false);
            while (t < m);
        } else {
            const int end = t < 64 && m > 64 ? 64 : last + 1;
            do GBA_W2_STEP(true);
            while (t < end);
        }
    }
#undef GBA_W2_STEP

    // Combine this lane's candidates, then the warp's, in the reference's order.
    Best1 best = w.bl;
    best.offer(w.bh.s, w.bh.e, w.bh.f, w.bh.col, w.bh.row);
    best.offer(row0.s, row0.e, row0.f, row0.col, row0.row);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int os = __shfl_down_sync(0xffffffffu, best.s, off);
        const int oe = __shfl_down_sync(0xffffffffu, best.e, off);
        const int of = __shfl_down_sync(0xffffffffu, best.f, off);
        const int oc = __shfl_down_sync(0xffffffffu, best.col, off);
        const int orr = __shfl_down_sync(0xffffffffu, best.row, off);
        if (lane + off < 32) best.offer(os, oe, of, oc, orr);
    }
    if (bands > 1 && seq) {
        if (lane == 0) carry.offer(best.s, best.e, best.f, best.col, best.row);
        if (b + 1 < bands) return;
        best = carry;
    } else if (bands > 1) {
        // Chain the bands' best cells in band order.
        if (b > 0) {
            warp_wait_at_least(&st[-1].done, 1, a.error);
            if (lane == 0) {
                const BandState *q = st - 1;
                best.offer(__ldcg(&q->s), __ldcg(&q->e), __ldcg(&q->f), __ldcg(&q->col), __ldcg(&q->row));
            }
        }
        if (b + 1 < bands) {
            if (lane == 0) {
                st->s = best.s;
                st->e = best.e;
                st->f = best.f;
                st->col = best.col;
                st->row = best.row;
                st_release_gpu(&st->done, 1);
            }
            return;
        }
    }
    if (lane == 0) {
        a.score[p] = best.s;
        if (a.end_h) a.end_h[p] = best.col;
        if (a.end_v) a.end_v[p] = best.row;
        if (a.best_e) a.best_e[p] = best.e;
        if (a.best_f) a.best_f[p] = best.f;
    }
}

template <bool AFFINE, bool LOCAL, int MAT, bool TRACE>
__global__ void __launch_bounds__(32 * kW2Warps, 4) k_dp_warp2(Warp2Args a)
{
    extern __shared__ uint2 profiles[];
    __shared__ int smat[MAT == W2_TABLE ? 32 * 32 : 1];
    __shared__ int8_t bmat[MAT == W2_PROFILE ? 32 * 32 : 1];
    if (MAT != W2_EQUAL) {
        for (int i = threadIdx.x; i < 32 * 32; i += blockDim.x) {
            const int r = i >> 5, c = i & 31;
            const int v = (r < a.alphabet && c < a.alphabet) ? a.matrix[r * a.alphabet + c] : 0;
            if (MAT == W2_TABLE) smat[i] = v;
            else bmat[i] = int8_t(v);
        }
    }
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    uint8_t *profile = nullptr;
    uint32_t outside = 0;
    if (MAT == W2_PROFILE) {
        profile = reinterpret_cast<uint8_t *>(profiles) + warp * w2_profile_bytes(a.alphabet);
        outside = uint32_t((kW2Warps - warp) * w2_profile_bytes(a.alphabet));
        if (threadIdx.x < 64) profiles[kW2Warps * w2_profile_bytes(a.alphabet) / 8 + threadIdx.x] = make_uint2(0, 0);
    }
    if (MAT != W2_EQUAL) __syncthreads();
    constexpr int kMost = MAT == W2_TABLE ? 4 : (LOCAL && TRACE ? 6 : 8);
    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(a.task_counter, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= a.num_tasks) break;
        const int2 pb = a.tasks[task];
        const PairDesc d = a.pairs[pb.x];
        const bool seq = pb.y < 0;
        Best1 carry{-(1 << 30), -(1 << 30), -(1 << 30), 0, 0};
        const int b0 = seq ? 0 : pb.y, b1 = seq ? w2_bands(d.n, d.rows) : pb.y + 1;
        for (int b = b0; b < b1; ++b) {
#define GBA_W2_BAND(R)                                                                                              \
    case R:                                                                                                         \
        if constexpr (R <= kMost)                                                                                   \
            warp2_band<AFFINE, LOCAL, MAT, TRACE, R>(a, smat, bmat, profile, outside, pb.x, b, lane, seq, carry);   \
        break
            switch (d.rows) {
                GBA_W2_BAND(2);
                GBA_W2_BAND(3);
                GBA_W2_BAND(4);
                GBA_W2_BAND(5);
                GBA_W2_BAND(6);
                GBA_W2_BAND(8);
            }
#undef GBA_W2_BAND
            __syncwarp();
        }
    }
}

}  // namespace gba
