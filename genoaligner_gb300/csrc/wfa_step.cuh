// wfa_step.cuh -- the wavefront recurrence and the walk of one pair on a group
// of G lanes (8, 16 or 32 of a warp, or the threads of a block), shared by the
// WFA kernels (wfa.cu, wfa_routed.cu, wfa_block.cu).  Recurrence and walk order
// are the reference's (include/genoaligner/backend/wfa_kernel.hip:119-145,
// 338-437; see wfa.cu).
#pragma once

#include "kernels.cuh"

namespace ga {

template <int G>
__device__ __forceinline__ void gsync(unsigned gmask)
{
    if (G > 32) __syncthreads();
    else if (G == 32) __syncwarp();
    else __syncwarp(gmask);
}

// A run of `len` copies of `c` ending just before slot[pos], its first byte
// `head` instead, written by the G lanes of a group; returns the new (lower)
// position.
template <int G>
__device__ __forceinline__ int emit_run_g(char* slot, int pos, int len, char c, char head, int gl, int* err)
{
    if (len <= 0) return pos;
    if (len > pos) {
        if (gl == 0) atomicOr(err, ERR_CIGAR_OVERFLOW);
        len = pos;
    }
    for (int q = gl; q < len; q += G) slot[pos - len + q] = q == 0 ? head : c;
    return pos - len;
}

// Length of the run of equal symbols of P from v and T from h, bounded by both
// ends.  2-bit codes: 16 at a time from 32-bit words (one funnel shift a side);
// the 64-bit window before it took four shifts a side and a 64-bit
// find-first-set, about twice the instructions, and off the main diagonal a run
// rarely passes its first base.  The kernels are bound by instruction issue: with
// this and one barrier a step, 20,000 pairs of 2 kb at smax 256, score only,
// 1.31 -> 0.66 ms.
template <int BITS>
__device__ __forceinline__ int extend_run(const uint64_t* __restrict__ P, const uint64_t* __restrict__ T, int v, int h,
                                          int m, int n)
{
    if constexpr (BITS != 2) {
        return match_run<BITS>(P, T, v, h, m, n);
    } else {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(P);
        const uint32_t* t = reinterpret_cast<const uint32_t*>(T);
        const int lim = min(m - v, n - h);
        int run = 0;
        while (run < lim) {
            const int a = (v + run) >> 4, b = (h + run) >> 4;
            const uint32_t x = __funnelshift_r(__ldg(p + a), __ldg(p + a + 1), 2 * (v + run)) ^
                               __funnelshift_r(__ldg(t + b), __ldg(t + b + 1), 2 * (h + run));
            if (x) { run += __clz((int)__brev(x)) >> 1; break; }
            run += 16;
        }
        return max(0, min(run, lim));
    }
}

// Wavefront value of diagonal k from the wavefront before (W at diagonal 0 of
// it): compute-next, clip past either end, extend.
template <int BITS>
__device__ __forceinline__ int next_offset(const int32_t* W, int k, const uint64_t* __restrict__ P,
                                           const uint64_t* __restrict__ T, int m, int n)
{
    const int x = max(W[k + 1], max(W[k - 1], W[k]) + 1);
    if ((unsigned)x > (unsigned)n || x - k > m) return WFA_NULL;        // (a dead offset is negative)
    return x + extend_run<BITS>(P, T, x - k, x, m, n);
}

// Wavefront values of diagonals k and k + G (the second where k + G <= hi; else it
// is WFA_NULL) on 2-bit codes: next_offset for both with their first 16 bases
// loaded together, so the two chains from wavefront to words to result overlap.
__device__ __forceinline__ void next_offsets2(const int32_t* W, int k, int k2, bool two, const uint64_t* __restrict__ P,
                                              const uint64_t* __restrict__ T, int m, int n, int& r0, int& r1)
{
    const uint32_t* p = reinterpret_cast<const uint32_t*>(P);
    const uint32_t* t = reinterpret_cast<const uint32_t*>(T);
    const int x0 = max(W[k + 1], max(W[k - 1], W[k]) + 1);
    const int x1 = two ? max(W[k2 + 1], max(W[k2 - 1], W[k2]) + 1) : WFA_NULL;
    const int lim0 = min(m - (x0 - k), n - x0), lim1 = min(m - (x1 - k2), n - x1);
    const bool live0 = (unsigned)x0 <= (unsigned)n && x0 - k <= m, live1 = (unsigned)x1 <= (unsigned)n && x1 - k2 <= m;
    const int v0 = live0 ? x0 - k : 0, h0 = live0 ? x0 : 0, v1 = live1 ? x1 - k2 : 0, h1 = live1 ? x1 : 0;
    const uint32_t a0 = __ldg(p + (v0 >> 4)), a1 = __ldg(p + (v0 >> 4) + 1), b0 = __ldg(t + (h0 >> 4)),
                   b1 = __ldg(t + (h0 >> 4) + 1);
    const uint32_t c0 = __ldg(p + (v1 >> 4)), c1 = __ldg(p + (v1 >> 4) + 1), d0 = __ldg(t + (h1 >> 4)),
                   d1 = __ldg(t + (h1 >> 4) + 1);
    const uint32_t e0 = __funnelshift_r(a0, a1, 2 * v0) ^ __funnelshift_r(b0, b1, 2 * h0);
    const uint32_t e1 = __funnelshift_r(c0, c1, 2 * v1) ^ __funnelshift_r(d0, d1, 2 * h1);
    int run0 = e0 ? __clz((int)__brev(e0)) >> 1 : 16, run1 = e1 ? __clz((int)__brev(e1)) >> 1 : 16;
    run0 = min(run0, lim0);
    run1 = min(run1, lim1);
    if (live0 && run0 == 16 && lim0 > 16) run0 += extend_run<2>(P, T, v0 + 16, h0 + 16, m, n);
    if (live1 && run1 == 16 && lim1 > 16) run1 += extend_run<2>(P, T, v1 + 16, h1 + 16, m, n);
    r0 = live0 ? x0 + run0 : WFA_NULL;
    r1 = live1 ? x1 + run1 : WFA_NULL;
}

// Diagonals of wavefront s that can matter: within reach of s edits, inside the
// matrix, and close enough to the final diagonal for the edits left up to smax.
// The values there are the full wavefront's: what they read of the one before
// lies in its range or holds NULL.
__device__ __forceinline__ int wave_lo(int s, int m, int kfinal, int smax) { return max(max(-s, -m), kfinal - (smax - s)); }
__device__ __forceinline__ int wave_hi(int s, int n, int kfinal, int smax) { return min(min(s, n), kfinal + (smax - s)); }

// The score of one pair on the G lanes of a group, -1 when it is above smax.
// wf0, wf1: 2 smax + 3 ints each; stk (trace): wavefront s at diagonal k goes to
// stk[s * s + s + k].  One barrier a step: a step reads the wavefront before and
// writes the other buffer, which the step before it was the last to read.
// AHEAD: two diagonals a lane at once (next_offsets2).  It shortens a lone pair's
// chain and lengthens the code: a batch of no more pairs than resident warps, bound
// by that chain, gains (the warps' 669 pairs of the 2,000-pair long batch: 1.0 ->
// 0.73 ms), a full device, bound by instruction issue, loses (20,000 x 2 kb: 656 ->
// 695 us).
// REACH: a pair above smax returns -1 less the offset it has reached on its final diagonal.
template <bool TRACE, int BITS, int G, bool AHEAD = false, bool REACH = false>
__device__ int wfa_forward(const uint64_t* __restrict__ P, const uint64_t* __restrict__ T, int m, int n, int smax,
                           int32_t* wf0, int32_t* wf1, int32_t* stk, int gl, unsigned gmask)
{
    const int kfinal = n - m;
    if (kfinal < -smax || kfinal > smax) return -1;
    const int WS = 2 * smax + 3;
    for (int t = gl; t < WS; t += G) { wf0[t] = WFA_NULL; wf1[t] = WFA_NULL; }
    const int off0 = extend_run<BITS>(P, T, 0, 0, m, n);
    if (kfinal == 0 && off0 >= n) return 0;
    gsync<G>(gmask);
    int32_t* prev = wf0 + smax + 1;                        // diagonal 0
    int32_t* cur = wf1 + smax + 1;
    if (gl == 0) {
        prev[0] = off0;
        if (TRACE) stk[0] = off0;
    }
    gsync<G>(gmask);
    [[maybe_unused]] int reach = 0;
    for (int s = 1; s <= smax; ++s) {
        const int hi = wave_hi(s, n, kfinal, smax);
        int32_t* const row = TRACE ? stk + (int64_t)s * s + s : nullptr;
        if constexpr (BITS == 2 && AHEAD) {
            for (int k = wave_lo(s, m, kfinal, smax) + gl; k <= hi; k += 2 * G) {
                const bool two = k + G <= hi;
                int x0, x1;
                next_offsets2(prev, k, k + G, two, P, T, m, n, x0, x1);
                cur[k] = x0;
                if (TRACE) row[k] = x0;
                if (two) {
                    cur[k + G] = x1;
                    if (TRACE) row[k + G] = x1;
                }
            }
        } else {
            for (int k = wave_lo(s, m, kfinal, smax) + gl; k <= hi; k += G) {
                const int x = next_offset<BITS>(prev, k, P, T, m, n);
                cur[k] = x;
                if (TRACE) row[k] = x;
            }
        }
        gsync<G>(gmask);
        if constexpr (REACH) {
            reach = cur[kfinal];
            if (reach >= n) return s;
        } else {
            if (cur[kfinal] >= n) return s;
        }
        int32_t* t = prev; prev = cur; cur = t;
    }
    if constexpr (REACH) return -1 - max(reach, 0);
    else return -1;
}

// The walk's choice at a cell from the wavefront before: the offset it came from
// and the op (mismatch on ties, then insertion, then deletion, strictly); 0 when
// none is live.
__device__ __forceinline__ char walk_choice(int w_mis, int w_ins, int w_del, int& best)
{
    const int c_mis = w_mis + 1, c_ins = w_ins + 1, c_del = w_del;
    best = WFA_NULL;
    char op = 0;
    if (wfa_live(c_mis) && c_mis >= best) { best = c_mis; op = 'X'; }
    if (wfa_live(c_ins) && c_ins > best)  { best = c_ins; op = 'I'; }
    if (wfa_live(c_del) && c_del > best)  { best = c_del; op = 'D'; }
    return op;
}

// The walk of a resolved pair (score >= 0) on the G lanes of its group, G <= 32,
// from the wavefront stack the forward pass left, written backwards from the end
// of the pair's CIGAR slot.  Every lane of the group runs the same walk; the runs
// are written by all of them.  The cells a step may read lie within one diagonal
// of where it stands, so the group loads those of the next R steps at once (rows
// of 3, 5, 7 ... offsets) and takes them by shuffles: one trip to memory every R
// steps of the walk's chain, not every step.  Returns the position of the
// CIGAR's first op in the slot.
template <int G>
__device__ int walk_g(const WfaArgs& A, int p, int score, int kfinal, int m, int n, const int32_t* stk, int gl,
                      unsigned gmask)
{
    char* slot = A.out_cigar + A.D.out_off[p];
    int pos = m + n;
    if (score == 0) return emit_run_g<G>(slot, pos, n, 'M', 'M', gl, A.err);
    constexpr int R = G >= 24 ? 4 : (G >= 15 ? 3 : 2);     // R (R + 2) offsets
    int u = 0;                                             // this lane's row of the next R, and its diagonal there
    while ((u + 1) * (u + 3) <= gl) ++u;
    const int c = gl - u * (u + 2) - (u + 1);
    int s = score, k = kfinal;
    int off = stk[(int64_t)s * s + s + k];
    int h = off, v = off - k;
    pos = emit_run_g<G>(slot, pos, v - m, 'D', 'D', gl, A.err);
    pos = emit_run_g<G>(slot, pos, h - n, 'I', 'I', gl, A.err);
    v = min(v, m);
    h = min(h, n);
    int w = WFA_NULL, row = R, dk = 0;
    while (v > 0 && h > 0 && s > 0) {
        if (row == R) {
            const int sp = s - 1 - u, kk = k + c;
            w = u < R && sp >= 0 && kk >= max(-sp, -m) && kk <= min(sp, n) ? stk[(int64_t)sp * sp + sp + kk] : WFA_NULL;
            row = 0;
            dk = 0;
        }
        const int at = row * (row + 2) + row + 1 + dk;
        const int w_mis = __shfl_sync(gmask, w, at, G), w_ins = __shfl_sync(gmask, w, at - 1, G);
        const int w_del = __shfl_sync(gmask, w, at + 1, G);
        int best;
        const char op = walk_choice(w_mis, w_ins, w_del, best);
        if (!op) break;
        pos = emit_run_g<G>(slot, pos, off - best + 1, 'M', op, gl, A.err);
        off = best;
        if (op == 'X')      { off -= 1; }
        else if (op == 'I') { k -= 1; dk -= 1; off -= 1; }
        else                { k += 1; dk += 1; }
        h = off;
        v = off - k;
        --s;
        ++row;
    }
    if (v > 0 && h > 0) {
        const int run = min(v, h);
        pos = emit_run_g<G>(slot, pos, run, 'M', 'M', gl, A.err);
        v -= run;
        h -= run;
    }
    pos = emit_run_g<G>(slot, pos, v, 'D', 'D', gl, A.err);
    return emit_run_g<G>(slot, pos, h, 'I', 'I', gl, A.err);
}

}  // namespace ga
