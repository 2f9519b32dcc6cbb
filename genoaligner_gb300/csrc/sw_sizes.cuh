// sw_sizes.cuh -- shapes, eligibility and per-warp memory of the
// Smith-Waterman traceback kernels, shared by the kernels (sw16ck.cu,
// sw32ck.cu), the device planner (sw_plan.cu) and the host.
#pragma once

#include <cmath>
#include <cstdint>

namespace ga {

// ---- 16-bit two-pairs-per-warp kernels --------------------------------------
// Every value is stored as value + BIAS16 so each 16-bit half stays in
// [0, 32767].  A pair qualifies when both sides hold only A, C, G, T and N and
// match * min(m, n) + BIAS16 + gap_open < 32000, gap_open + gap_extend < BIAS16
// and mismatch + gap_open >= 0 (host-side check; purity comes from the device).
constexpr int BIAS16 = 1024;

__host__ __device__ inline bool sw16_eligible(int m, int n, int match, int mismatch, int go, int ge)
{
    if (m <= 0 || n <= 0) return false;
    if (go + ge >= BIAS16 || mismatch + go < 0 || match + go > 32000) return false;
    const int64_t top = (int64_t)match * (m < n ? m : n) + BIAS16 + go;
    return top < 32000;
}

// The 16-bit traceback kernel keeps a row number in 16 bits: longer texts are the
// 32-bit kernels'.
constexpr int SW16_TRACE_ROWS = 65535;

// Optimistic 16-bit eligibility: the bound above with the all-match score
// scaled by pct / 100 (pct 100: the bound itself).  A pair taken on this
// rule alone may score past 16 bits; the kernel then sees a best value of at
// least sw16_overflow_limit and hands the pair to the 32-bit kernel.
__host__ __device__ inline bool sw16_eligible_opt(int m, int n, int match, int mismatch, int go, int ge, int pct)
{
    if (m <= 0 || n <= 0) return false;
    if (go + ge >= BIAS16 || mismatch + go < 0 || match + go > 32000) return false;
    const int64_t top = (int64_t)match * (m < n ? m : n) * pct / 100 + BIAS16 + go;
    return top < 32000;
}

// The scheme conditions of the 16-bit kernels alone (no score bound): the
// per-pair 16-bit choice of the SW model is taken only under them.
__host__ __device__ inline bool sw16_scheme_ok(int match, int mismatch, int go, int ge)
{
    return go + ge < BIAS16 && mismatch + go >= 0 && match + go <= 32000;
}

// A best value at or above this in the 16-bit forward pass may have passed
// 16 bits somewhere: every cell's value is exact until an H_diag + match
// first wraps, and that H_diag (> 32767 - match) is in the best, so a best
// below the limit proves the whole pass (and the biased windows, values up to
// best + BIAS16 + match) exact.
__host__ __device__ inline int sw16_overflow_limit(int match) { return 32000 - BIAS16 - match; }

// sw16ck.cu: checkpoint rows every CK_K rows, column edges every CK_TW
// columns, recompute windows of `window` tiles of CK_K x CK_TW cells (2 or 4;
// CK_TG is the default).
constexpr int CK_K = 64;
constexpr int CK_TW = 64;
constexpr int CK_TG = 2;
constexpr int CK_C = 16;                 // forward columns per lane, full bands
constexpr int CK_BW = 32 * CK_C;         // forward band width, full bands

__host__ __device__ inline int ck_rows(int M) { return M > 1 ? (M - 1) / CK_K : 0; }

// Forward bands: full bands of CK_BW columns while more than CK_BW columns
// remain, then one band of 32 * CB columns with the smallest CB in
// {2, 4, 8, 16} that reaches column N.
__host__ __device__ inline int ck_last_cb(int rest)
{
    return rest > 8 * 32 ? 16 : (rest > 4 * 32 ? 8 : (rest > 2 * 32 ? 4 : 2));
}
// Columns the forward bands cover (the column extent of the checkpoints).
__host__ __device__ inline int ck_ncol(int N)
{
    const int full = N > 0 ? (N - 1) / CK_BW : 0;
    return full * CK_BW + 32 * ck_last_cb(N - full * CK_BW);
}

// 32-bit words of one warp slot for an item of at most M rows and N columns:
// checkpoint rows, column edges (16-byte aligned end), the window table.
__host__ __device__ inline int64_t sw16ck_dir_words(int M, int N, int window)
{
    const int64_t ncol = ck_ncol(N);
    return 2 * (int64_t)ck_rows(M) * ncol + (2 * (ncol / CK_TW) * (int64_t)M + 3) / 4 * 4 +
           (int64_t)CK_K * window * CK_TW;
}

// A 16-bit pair of n columns is listed by its cells, before those that are not.
__host__ __device__ inline bool sw16_by_cells(int n) { return ck_ncol(n > 1 ? n : 1) >= 24 * 64; }

// Bucket (0..4095, smallest first) of a 16-bit pair of m rows and n columns
// in a list of the two-pairs-per-warp kernels: consecutive entries share a
// warp and run with the larger of their row counts and forward column
// extents, so the key orders by column extent (ck_ncol, in 64-column steps,
// widest first), then by rows (18 buckets per doubling, most first):
// neighbours then have near-equal shapes, not only near-equal cell counts.
// Pairs 1,536 columns wide and more come before all others, by cells (32
// buckets per doubling, largest first), so the longest work starts first and
// whole-block items lead.
__host__ __device__ inline int sw16_shape_key(int m, int n)
{
    const int ncls = ck_ncol(n > 1 ? n : 1) / 64;
    if (sw16_by_cells(n)) {
        const float lc = log2f((float)(m > 1 ? m : 1) * (float)(n > 1 ? n : 1));
        const int e = (int)(32.0f * (lc - 20.0f));
        return 1023 - (e < 0 ? 0 : (e > 1023 ? 1023 : e));
    }
    const float lm = log2f((float)(m > 16 ? m : 16) * (1.0f / 16.0f));
    const int mb = (int)(18.0f * lm) < 127 ? (int)(18.0f * lm) : 127;
    return 1024 + (23 - ncls) * 128 + (127 - mb);
}

// 32-bit words of one warp slot of the 16-bit score-only kernel (sw16so in
// sw16ck.cu): per pair and lane the row that last raised the lane's best
// (SO_ROW_WORDS), then the column edges that carry its band boundaries.
constexpr int SO_ROW_WORDS = 2 * 32 * CK_C;
__host__ __device__ inline int64_t sw16so_dir_words(int M, int N)
{
    return SO_ROW_WORDS + (2 * (int64_t)(ck_ncol(N) / CK_TW) * M + 3) / 4 * 4 + 4;
}

// Items of a traceback list above this many cells run on a whole block: above
// limit (the sw_coop_log2 setting, < 0: none), and above twice the list's cells per
// resident warp.  An item past that share would keep its one warp busy when the
// others have run out of work: 152 pairs of 8,000 x 8,000 take 28.8 ms on a warp
// each and 5.2 ms on a block each, and batches with more items than warps stay
// below the share.  Items under SW_COOP_MIN cells have too few bands to divide.
constexpr int64_t SW_COOP_MIN = (int64_t)1 << 16;
__host__ __device__ inline int64_t sp_coop_cells(int64_t limit, int64_t cells, int64_t warps)
{
    if (limit < 0 || warps <= 0) return INT64_MAX;
    const int64_t share = 2 * cells / warps;
    const int64_t t = share < SW_COOP_MIN ? SW_COOP_MIN : share;
    return t < limit ? t : limit;
}
// Near-equal items, too many for that: a cell costs a block's warps 1.8 times what it
// costs a multiprocessor full of single ones, so a list that gives every multiprocessor
// some six items and more, none above 1.6 times the mean, stays on warps whatever their
// share.  (32 bits, on blocks and on warps: 900 pairs of 800 x 850 1,647 and 1,714
// us, 1,000 1,896 and 1,733, 1,200 2,169 and 1,779; 1,000 of 3,100 x 3,200 7.7 and 9.1 ms,
// 1,100 12.1 and 9.3.  16 bits: 1,000 items of 1,400 x 1,500 3.11 and 2.95 ms, 1,150
// 4.43 and 2.88; 1,000 of 3,100 x 3,200 9.8 and 10.3, 1,150 13.5 and 10.1.)
__host__ __device__ inline bool sw_even_many(int64_t items, int64_t largest, int64_t cells, int cols, int64_t warps)
{
    return 5 * largest * items <= 8 * cells && 40 * items > (cols >= 2048 ? 17 : 15) * warps;
}
// Warps of a whole-block launch's blocks, 4, 8 or 16: enough that the largest item,
// which gets W of a multiprocessor's 16 resident warps, ends no later than the
// multiprocessors' common work, and no more than a quarter of the 64-column bands it
// can be cut into.  (With the walk still one warp's, 152, 304 and 608 pairs of 8,000 x
// 8,000 took 11.4, 13.1, 21.2 ms with 4 warps, 8.9, 12.2, 24.6 with 8, 8.2, 16.2, 32.2
// with 16; 1,024 pairs of 2 to 30 kb, one of them 1/150 of the cells, 280, 217, 153 ms;
// 600 pairs of 200 to 1,000 x 1,100 score-only 0.61, 0.71, 1.54 ms.)
constexpr int COOP_MAX_WARPS = 16;
__host__ __device__ inline int sw_coop_block(int64_t largest, int cols, int64_t cells, int sms)
{
    int W = 4;
    while (W < COOP_MAX_WARPS && W * 512 <= cols && W * cells < 16 * largest * sms) W *= 2;
    return W;
}
// Per-warp share of an item's memory when a block of W warps serves it, `own` words
// of it for each warp: the score-only kernel's rows, the traceback kernels' table.
__host__ __device__ inline int64_t sw_coop_share(int64_t words, int W, int64_t own = 0)
{
    return own + (words - own + 4 * W - 1) / (4 * W) * 4;
}
__host__ __device__ inline int64_t sw16_own_words(bool trace, int window)
{
    return trace ? (int64_t)CK_K * window * CK_TW : SO_ROW_WORDS;
}
// Columns per lane of a whole-block item's full bands: those of 16, 8 and down to
// `least` with the shortest schedule, of start(last band) + chunks chunks (fwd16_coop)
// of CB + 4 units each.
__host__ __device__ inline int coop_cb(int N, int W, int nck, int least)
{
    int best = 16;
    int64_t t = INT64_MAX;
    for (int cb = 16; cb >= least; cb >>= 1) {
        const int last = (N - 1) / (32 * cb);
        const int64_t g = (int64_t)(last / W) * (nck > 2 * W ? nck : 2 * W) + 2 * (last % W) + nck;
        if (g * (cb + 4) < t) { t = g * (cb + 4); best = cb; }
    }
    return best;
}

// ---- 32-bit one-pair-per-warp checkpointed kernel (sw32ck.cu) ---------------
constexpr int C32_C = 16;                // forward columns per lane, full bands
constexpr int C32_BW = 32 * C32_C;
constexpr int C32_LONG_LOG2 = 24;       // default: the long-pair shape above 2^24 cells
constexpr int C32_COOP_LOG2 = 27;       // default: work items above 2^27 cells run on a whole block

__host__ __device__ inline int c32_rows(int m, int K) { return m > 1 ? (m - 1) / K : 0; }
__host__ __device__ inline int c32_last_cb(int rest) { return rest > 8 * 32 ? 16 : (rest > 4 * 32 ? 8 : 4); }
__host__ __device__ inline int c32_ncol(int n)
{
    const int full = n > 0 ? (n - 1) / C32_BW : 0;
    return full * C32_BW + 32 * c32_last_cb(n - full * C32_BW);
}
// The long-pair shape (512-row blocks, 512-column tiles) for pairs above
// 2^long_log2 cells, the short one (64 x 64) below.
__host__ __device__ inline bool sw32ck_long(int m, int n, int long_log2)
{
    return (int64_t)m * n > ((int64_t)1 << long_log2);
}

// 32-bit words of one warp slot for a pair of m rows and n columns:
// checkpoint rows, column edges, the tile table.
__host__ __device__ inline int64_t sw32ck_dir_words(int m, int n, int long_log2)
{
    const bool lg = sw32ck_long(m, n, long_log2);
    const int K = lg ? 512 : 64, CT = lg ? 16 : 2, TW = 32 * CT, NWT = CT >= 8 ? CT / 8 : 1;
    const int64_t stride = ((int64_t)c32_ncol(n) + TW - 1) / TW * TW;
    return 2 * (int64_t)c32_rows(m, K) * stride + 2 * (stride / TW) * (int64_t)m + (int64_t)(K + 31) * 32 * NWT;
}

// The tile table's part of them (sw_coop_share's own words).
__host__ __device__ inline int64_t sw32_own_words(int m, int n, int long_log2)
{
    return sw32ck_long(m, n, long_log2) ? (512 + 31) * 32 * 2 : (64 + 31) * 32;
}

}  // namespace ga
