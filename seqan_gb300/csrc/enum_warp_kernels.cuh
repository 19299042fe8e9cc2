// enum_warp_kernels.cuh -- Waterman-Eggert enumeration (enum_kernels.cuh), a warp per pair.
//
// The enumeration's order of events is the reference's, one after the other; what a warp does at
// once is the inside of each event:
//   * fill: the matrix as a wavefront of 32 rows.  The cells >= cutoff are then pushed in the
//     reference's scan order.
//   * push: the lanes read all ancestors of the new leaf in one access; those below the pushed
//     score are the first ones of the path, and each moves to its child.
//   * toward the leaves: the path of larger children (the left one of equals) does not depend on
//     the entry that sinks, only its end does.  A bit per inner node says which child is the larger, so
//     the path to the bottom is three words of five levels; the lanes then read all its nodes and their
//     siblings in one access, each node above the entry moves to its parent, and where it is no longer
//     above its sibling its parent's bit turns.
//   * declump: a row's cells right to left, 32 at a time; the chain of horizontal gaps is a
//     max-plus scan that a match (which takes its diagonal whatever else scores) starts anew.  The
//     rules that end a row and move its right end are prefixes of the lanes' comparisons.
//
// Scores of up to 15 bits and matrices of up to 2^16 cells: a heap entry is one word (score,
// position), a matrix cell 15 bits and the forbidden flag, the larger-child bits 4 KB of shared memory.
//
// Bound by latency and issue alike: an enumeration refreshes thousands of stale entries one after
// the other (7,000 of 18,000 at 150 bp, ten alignments), each one dependent miss and about 100 instructions,
// and a pair's heap (70 KB) and matrix (45 KB) are far beyond its share of the caches.  10,000 pairs of
// 100-200 bp, half related, 2/-1/-2, cutoff 10, ten alignments: 31.5 ms, one thread per pair 138.5.
// Steps on the way: the path four levels at a time from the nodes themselves, without bits, 42; scratch
// per pair instead of per resident warp 49; eight blocks an SM (64 registers) 31.5, six 32.6, ten 38.4.
#pragma once

#include "enum_kernels.cuh"

namespace gba {

constexpr int kWeBits = 1 + 32 + 1024;   // words of larger-child bits: subtrees of five levels at depths 0, 5, 10
constexpr int kWeTop = 1024;             // heap nodes below this are in shared memory during the fill
constexpr int kWeSteps = 1024;           // most steps of a trace (m + n)
constexpr int kWePosBits = 16;
constexpr uint32_t kWePos = (1u << kWePosBits) - 1;
constexpr int kWeWarps = 4;              // warps of a block

struct WeWarpArgs {
    EnumArgs e;                       // mat, forb, heap and steps unused
    const int32_t *order;             // pairs, the largest first (null: as they come)
    // Per resident warp: heap of m * n + 2 nodes (1-based), then the matrix of (m + 1) * (n + 1) cells
    // (value, bit 15 forbidden), for the largest of the pairs.
    uint8_t *scratch;
    int64_t stride, mat_at;
    int32_t *next;                    // work counter
};

// Per warp: the larger-child bits, then the trace's steps.
extern __shared__ uint32_t we_shared[];
constexpr int kWeWords = kWeBits + kWeSteps / 4;

struct WeWarp {
    const EnumArgs &a;
    int32_t base;                     // the warp's part of we_shared
    int32_t lane;
    const uint8_t *H, *V;
    uint16_t *M;
    uint32_t *hp;                     // heap nodes, 1-based
    int32_t m, n, W, hn;
    int32_t T, x0, y0, endH, endV, best_end, best_begin;

    __device__ __forceinline__ int sc(int x, int y) const
    {
        if (a.matrix) return a.matrix[x * a.alphabet + y];
        return x == y ? a.match : a.mismatch;
    }
    // steps of the trace (bit 0: consumes H, bit 1: consumes V), behind the heap's first nodes
    __device__ __forceinline__ uint8_t &step(int t) const { return reinterpret_cast<uint8_t *>(we_shared + base + kWeBits)[t]; }
    __device__ __forceinline__ int value(int pos) const { return M[pos] & 0x7fff; }
    // push + _adjustHeapTowardRoot.  Lane k holds the k-th ancestor of the new leaf; the first c are
    // below e, each moves to its child's place and e takes the c-th one's.  While the heap is filled its
    // first nodes stand where the bits will.
    __device__ __forceinline__ void push(uint32_t e)
    {
        const int up = ++hn >> lane;                        // (hn < 2^16: lanes 16 .. 31 have none)
        uint32_t *const at = (up < kWeTop ? we_shared + base : hp) + up;
        uint32_t v = 0xffffffffu;
        if (up > 0 && lane > 0) v = *at;
        const uint32_t below = __ballot_sync(0xffffffffu, v < (e & ~kWePos)) | 1u;
        const int c = 31 - __clz(int(below & ~(below + 1)));            // the run of ones from bit 0
        const uint32_t down = __shfl_down_sync(0xffffffffu, v, 1);
        if (lane <= c) *at = lane == c ? e : down;
        __syncwarp();
    }

    // The larger-child bit of inner node j, `above` levels below its subtree's root: word and bit.
    static __device__ __forceinline__ void bit_of(int j, int depth, int &word, uint32_t &bit)
    {
        const int above = depth % 5, r = j >> above;
        word = depth < 5 ? 0 : (depth < 10 ? r - 31 : r - 991);
        bit = 1u << (j + ((1 - r) << above));
    }

    // All bits, a subtree's 31 inner nodes at a time.
    __device__ void larger_children()
    {
        for (int j = 1 + lane; j < kWeTop && j <= hn; j += 32) hp[j] = we_shared[base + j];
        __syncwarp();
        const int depth = 31 - __clz(lane | 1);
        for (int word = 0; word < kWeBits; ++word) {
            const int root = word == 0 ? 1 : (word < 33 ? word + 31 : word + 991);
            if (2 * root > hn) {
                if (word == 0) continue;
                word = word < 33 ? 32 : kWeBits;            // the rest of this depth has no children
                continue;
            }
            const int j = (root << depth) + lane - (1 << depth);
            uint32_t x = 0, y = 0;
            if (lane > 0 && 2 * j <= hn) x = hp[2 * j];
            if (lane > 0 && 2 * j < hn) y = hp[2 * j + 1];
            const uint32_t bits = __ballot_sync(0xffffffffu, (x | kWePos) < y);
            if (lane == 0) we_shared[base + word] = bits;
        }
        __syncwarp();
    }

    // _adjustHeapTowardLeaves from the root; returns the new root and reads its cell's value.
    __device__ __forceinline__ uint32_t sink(uint32_t e, int *next_value)
    {
        const uint32_t above = e | kWePos;                  // v > above: v's score is the higher
        uint32_t w = we_shared[base];
        int leaf = 1;
        // the new root, and its cell's value ahead of its use
        const int child = 2 + int(w >> 1 & 1u);
        uint32_t top = child <= hn ? hp[child] : 0u;
        top = top > above ? top : e;
        *next_value = M[top & kWePos];
#pragma unroll
        for (int q = 0; q < 5; ++q) leaf = 2 * leaf + int(w >> leaf & 1u);
#pragma unroll
        for (int stage = 0; stage < 2; ++stage) {
            w = we_shared[base + leaf - (stage ? 991 : 31)];
            int l = 1;
#pragma unroll
            for (int q = 0; q < 5; ++q) l = 2 * l + int(w >> l & 1u);
            leaf = 32 * leaf + l - 32;
        }
        // lane k: the path's node at depth k
        const int j = leaf >> (15 - min(lane, 15));
        uint32_t v = 0, sibling = 0;
        if (lane < 16 && j <= hn) v = hp[j];
        if (lane < 16 && (j ^ 1) <= hn) sibling = hp[j ^ 1];
        const int c = __popc(__ballot_sync(0xffffffffu, lane > 0 && v > above));
        const uint32_t down = __shfl_down_sync(0xffffffffu, v, 1);
        const uint32_t now = lane == c ? e : down;
        if (lane <= c) hp[j] = now;
        // the larger child no more?
        if (lane > 0 && lane <= c && (j & 1 ? now <= (sibling | kWePos) : sibling > (now | kWePos))) {
            int word;
            uint32_t bit;
            bit_of(j >> 1, lane - 1, word, bit);
            atomicXor(&we_shared[base + word], bit);
        }
        __syncwarp();
        *next_value &= 0x7fff;
        return top;
    }

    // The last leaf, taken off the heap.
    __device__ __forceinline__ uint32_t last_leaf()
    {
        const uint32_t e = hp[hn];
        if (lane == 0 && hn > 1 && (hn & 1)) {              // its parent keeps a left child
            int word;
            uint32_t bit;
            bit_of(hn >> 1, 31 - __clz(hn >> 1), word, bit);
            we_shared[base + word] &= ~bit;
        }
        --hn;
        __syncwarp();
        return e;
    }

    // _smithWatermanGetMatrix (:112-175)
    __device__ void fill()
    {
        for (int x = lane; x <= m; x += 32) M[x + n * W] = 0;
        for (int y = lane; y <= n; y += 32) M[m + y * W] = 0;
        __syncwarp();
        for (int yb = n - 1; yb >= 0; yb -= 32) {
            const int y = yb - lane;
            const int cy = y >= 0 ? V[y] : 0;
            int v = 0, below_old = 0, chunk = 0;
            for (int t = 0; t < m + 31; ++t) {
                if ((t & 31) == 0) {                        // the row below the band, 32 cells ahead
                    const int x = m - 1 - t - lane;
                    chunk = x >= 0 ? M[x + (yb + 1) * W] & 0x7fff : 0;
                }
                int below = __shfl_up_sync(0xffffffffu, v, 1);
                const int first = __shfl_sync(0xffffffffu, chunk, t & 31);
                if (lane == 0) below = first;
                const int x = m - 1 - t + lane;
                if (y >= 0 && x >= 0 && x < m) {
                    const int hx = H[x], cs = sc(hx, cy);
                    if (hx == cy) v = below_old + cs;
                    else v = max(max(below_old + cs, a.gap + max(below, v)), 0);
                    M[x + y * W] = uint16_t(v);
                    below_old = below;
                }
            }
            __syncwarp();
        }
        for (int y = n - 1; y >= 0; --y)
            for (int xb = m - 1; xb >= 0; xb -= 32) {
                const int x = xb - lane, pos = x + y * W;
                const int v = x >= 0 ? M[pos] & 0x7fff : 0;
                uint32_t q = __ballot_sync(0xffffffffu, x >= 0 && v >= a.cutoff);
                const uint32_t e = uint32_t(v) << kWePosBits | (uint32_t(pos) & kWePos);
                while (q) {
                    push(__shfl_sync(0xffffffffu, e, __ffs(int(q)) - 1));
                    q &= q - 1;
                }
            }
    }

    // _smithWatermanTrace (:300-371)
    __device__ void trace(int src)
    {
        int i0 = src % W, i1 = src / W, t = 0;
        x0 = i0;
        y0 = i1;
        while (i0 != m && i1 != n) {
            const int here = M[src], right = M[src + 1] & 0x7fff, under = M[src + W] & 0x7fff,
                      cross = M[src + 1 + W] & 0x7fff, hx = H[i0], cy = V[i1];
            if ((here & 0x7fff) == 0) break;
            const bool forb = here >> 15;
            bool gv = true, gh = true;
            if (hx != cy || forb) {
                const int vr = right + a.gap, d = forb ? 0 : cross + sc(hx, cy), hd = under + a.gap;
                gv = (vr >= hd) | (d >= hd);
                gh = (hd > vr) | (d >= vr);
            }
            if (lane == 0) step(t) = uint8_t(gv | gh << 1);
            if (gv) { ++i0; src += 1; }
            if (gh) { ++i1; src += W; }
            ++t;
        }
        T = t;
        endH = i0;
        endV = i1;
        best_begin = src;
        __syncwarp();
    }

    // _smithWatermanDeclump (:176-299); false where the reference's walk leaves its arrays.
    __device__ bool declump()
    {
        // the first step that consumes H, and V
        int s0 = 0, s1 = 0;
        while (s0 < T && !(step(s0) & 1)) ++s0;
        while (s1 < T && !(step(s1) & 2)) ++s1;
        int a0 = T, a1 = T, forb = best_begin, xe = endH - 1, x_stop = xe;
        bool forbidden_reached = true, end_reached = false, skip_row = false;
        for (int y = endV - 1; y != -1; --y) {
            if (forbidden_reached && !end_reached) {
                if (a0 == s0 && a1 == s1) end_reached = true;
                if (!end_reached) {
                    --a0;
                    forb -= W;
                    if (x0 + a0 < 0 || y0 + a1 < 0 || forb < 0) return false;
                    while (a0 >= 0 && !(step(a0) & 1) && a0 != s0) {
                        skip_row = true;
                        --a0;
                        --a1;
                        forb -= W;
                        if (x0 + a0 < 0 || y0 + a1 < 0 || forb < 0) return false;
                    }
                    --a1;
                    forb -= 1;
                    if (x0 + a0 < 0 || y0 + a1 < 0 || forb < 0) return false;
                    while (a1 >= 0 && !(step(a1) & 2) && a1 != s1) {
                        --a1;
                        --a0;
                        forb -= 1;
                        if (x0 + a0 < 0 || y0 + a1 < 0 || forb < 0) return false;
                    }
                    if (lane == 0) M[forb] |= 0x8000;
                    __syncwarp();
                    forbidden_reached = false;
                }
            }
            const int cy = V[y];
            const int at = forb - y * W, fx = at >= 0 && at <= m ? at : -1;   // the forbidden cell in this row
            const bool shrink = !forbidden_reached && !skip_row;
            const int stop0 = x_stop, end0 = xe;
            int carry = value(end0 + 1 + y * W);
            bool leading = true;                            // no cell of this row has stayed at the right end
            for (int xb = end0; xb >= 0; xb -= 32) {
                const int x = xb - lane, pos = x + y * W;
                int old = 0, c = 0;
                bool match = false;
                if (x >= 0) {
                    old = M[pos];
                    const int diag = M[pos + W + 1] & 0x7fff, below = M[pos + W] & 0x7fff, hx = H[x];
                    const bool f = old >> 15;
                    const int cs = sc(hx, cy);
                    match = hx == cy && !f;
                    c = match ? diag + cs : max(max(f ? 0 : diag + cs, a.gap + below), 0);
                }
                const uint32_t B = __ballot_sync(0xffffffffu, match) & (0xffffffffu >> (31 - lane));
                const int reach = B ? lane - (31 - __clz(int(B))) : 32;    // lanes back to the chain's start
                int v = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o && o <= reach) v = max(v, t + o * a.gap);
                }
                if (reach == 32) v = max(v, carry + (lane + 1) * a.gap);
                const bool same = (old & 0x7fff) == v;
                const uint32_t S = __ballot_sync(0xffffffffu, x >= 0 && x < stop0 && same);
                const int visited = S ? __ffs(int(S)) : min(32, xb + 1);
                if (lane < visited) M[pos] = uint16_t(v | (old & 0x8000));
                if (leading) {
                    const uint32_t A = __ballot_sync(0xffffffffu, x >= 0 && same && x >= stop0 &&
                                                                      (end_reached || (shrink && x > fx)));
                    const int lead = A == 0xffffffffu ? 32 : __ffs(int(~A)) - 1;
                    xe -= lead;
                    leading = lead == 32;
                }
                if (fx <= xb && fx > xb - visited) {
                    skip_row = false;
                    forbidden_reached = true;
                }
                x_stop = min(x_stop, xb - visited + 1);
                carry = __shfl_sync(0xffffffffu, v, 31);
                if (S) break;
            }
            __syncwarp();
            if (xe == -1) break;
        }
        return true;
    }

    // _getNextBestEndPosition (:372-403), its pop left to the caller: entries whose cell has changed since
    // are entered anew, or dropped, until the root's has not.  The root, or 0 (hn == 0).
    __device__ __forceinline__ uint32_t next_end()
    {
        if (hn == 0) return 0;
        uint32_t root = hp[1];
        int top = value(int(root & kWePos));
        while (int(root >> kWePosBits) != top) {
            uint32_t e = uint32_t(top) << kWePosBits | (root & kWePos);
            if (top < a.cutoff) {
                e = last_leaf();
                if (hn == 0) return 0;
            }
            root = sink(e, &top);
        }
        return root;
    }

    __device__ __forceinline__ void pop()
    {
        const uint32_t e = last_leaf();
        int unused;
        if (hn > 0) sink(e, &unused);
    }
};

__global__ void __launch_bounds__(32 * kWeWarps, 8) k_waterman_eggert_warp(WeWarpArgs a)
{
    WeWarp w{a.e, int(threadIdx.x >> 5) * kWeWords, int(threadIdx.x & 31u)};
    uint8_t *const scratch = a.scratch + (int64_t(blockIdx.x) * kWeWarps + (threadIdx.x >> 5)) * a.stride;
    w.hp = reinterpret_cast<uint32_t *>(scratch);
    w.M = reinterpret_cast<uint16_t *>(scratch + a.mat_at);
    for (;;) {
        int p = 0;
        if (w.lane == 0) p = atomicAdd(a.next, 1);
        p = __shfl_sync(0xffffffffu, p, 0);
        if (p >= a.e.num_pairs) return;
        if (a.order) p = a.order[p];
        const EnumPair d = a.e.pairs[p];
        w.H = a.e.seq_h + d.h_off;
        w.V = a.e.seq_v + d.v_off;
        w.m = d.m;
        w.n = d.n;
        w.W = d.m + 1;
        w.hn = 0;
        int k = 0, status = 0;
        if (d.m > 0 && d.n > 0) {
            w.fill();
            w.larger_children();
            for (; k < a.e.max_count; ++k) {
                if (k > 0 && !w.declump()) {
                    status = 1;
                    break;
                }
                const uint32_t root = k > 0 ? w.next_end() : (w.hn > 0 ? w.hp[1] : 0u);
                if (w.hn == 0) break;
                w.best_end = int(root & kWePos);
                // (the reference takes position 0 for none, but not in its first alignment)
                if ((k > 0 && w.best_end == 0) || w.value(w.best_end) == 0) break;
                w.pop();
                w.trace(w.best_end);
                if (w.lane == 0) {
                    const int64_t o = int64_t(p) * a.e.max_count + k;
                    a.e.score[o] = w.value(w.best_end);
                    a.e.begin_h[o] = w.x0;
                    a.e.begin_v[o] = w.y0;
                    a.e.end_h[o] = w.endH;
                    a.e.end_v[o] = w.endV;
                    // the columns as runs in alignment order
                    uint4 *out = reinterpret_cast<uint4 *>(a.e.seg_slots) + d.seg_off + int64_t(k) * (d.m + d.n + 1);
                    int ns = 0, nextH = w.x0, nextV = w.y0;
                    for (int t = 0; t < w.T;) {
                        const int type = w.step(t);
                        int u = t + 1;
                        while (u < w.T && w.step(u) == type) ++u;
                        out[ns++] = make_uint4(uint32_t(nextH), uint32_t(nextV), uint32_t(u - t),
                                               type == 3 ? uint32_t(TV_DIAG) : (type == 1 ? uint32_t(TV_H) : uint32_t(TV_V)));
                        if (type & 1) nextH += u - t;
                        if (type & 2) nextV += u - t;
                        t = u;
                    }
                    a.e.seg_count[o] = ns;
                }
                __syncwarp();
            }
        }
        if (w.lane == 0) {
            a.e.count[p] = k;
            a.e.status[p] = status;
        }
        __syncwarp();
    }
}

}  // namespace gba
