// wfa_block.cu -- WFA pairs of large distance, each on a whole block.
//
// A pair at distance d is d dependent steps over up to 2 d + 1 diagonals: on one
// warp the largest pair of a batch sets its time.  Here the 512 threads of a
// block split a step's diagonals, with one block barrier a step (wfa_forward),
// and the block holds one pair's two wavefronts in shared memory -- 33 KB at
// smax 2048, so two blocks share an SM where the warp kernels, sized for one
// pair per warp at the batch smax, fitted a single block of four warps.  2,000
// pairs of 1-10 kb at smax 2048 with CIGARs: 9.6 ms of warp-queue kernel with
// blocks of 128 threads, 4.2 ms with these blocks and the warps' cap.
//
// Items: the router's pairs estimated at s >= 256 (largest first), then the
// pairs the warp kernels left unresolved at their last cap.
#include "wfa_step.cuh"

namespace ga {

constexpr int BLK_T = 512;               // threads per block
constexpr int BLK_ROWS = 15;             // wavefronts a walk loads at once ...
constexpr int BLK_ROW = 2 * (BLK_ROWS + 1) + 2;          // ... and the words of each (diagonals -16 .. 17)
static_assert(BLK_ROWS * BLK_ROW <= BLK_T, "a thread per word");

// The walk of a resolved pair (score > 0): the block loads the cells that the
// next BLK_ROWS steps may read into `buf`, its first warp takes those steps and
// writes their ops (walk_g's step).  Returns (to the first warp) the position
// of the CIGAR's first op in the slot.
__device__ int walk_block(const WfaArgs& A, int p, int score, int kfinal, int m, int n, const int32_t* stk, int32_t* buf,
                          int* s_at)
{
    const int t = threadIdx.x, lane = t & 31;
    char* slot = A.out_cigar + A.D.out_off[p];
    int pos = m + n, s = score, k = kfinal;
    int off = stk[(int64_t)s * s + s + k];
    int h = off, v = off - k;
    if (t < 32) {
        pos = emit_run_g<32>(slot, pos, v - m, 'D', 'D', lane, A.err);
        pos = emit_run_g<32>(slot, pos, h - n, 'I', 'I', lane, A.err);
    }
    v = min(v, m);
    h = min(h, n);
    const int u = t / BLK_ROW, c = t % BLK_ROW - (BLK_ROWS + 1);
    for (;;) {
        // (s, k) is the whole block's
        if (t < BLK_ROWS * BLK_ROW) {
            const int sp = s - 1 - u, kk = k + c;
            const bool in = c >= -(u + 1) && c <= u + 1 && sp >= 0 && kk >= max(-sp, -m) && kk <= min(sp, n);
            buf[t] = in ? stk[(int64_t)sp * sp + sp + kk] : WFA_NULL;
        }
        __syncthreads();
        if (t < 32) {
            bool more = true;
            int at = BLK_ROWS + 1;                         // buf word of diagonal k in the next row
            for (int r = 0; r < BLK_ROWS; ++r, at += BLK_ROW) {
                int best = 0;
                char op = 0;
                if (v > 0 && h > 0 && s > 0) op = walk_choice(buf[at], buf[at - 1], buf[at + 1], best);
                if (!op) { more = false; break; }
                pos = emit_run_g<32>(slot, pos, off - best + 1, 'M', op, lane, A.err);
                off = best;
                if (op == 'X')      { off -= 1; }
                else if (op == 'I') { k -= 1; at -= 1; off -= 1; }
                else                { k += 1; at += 1; }
                h = off;
                v = off - k;
                --s;
            }
            if (lane == 0) { s_at[0] = s; s_at[1] = k; s_at[2] = more; }
        }
        __syncthreads();
        s = s_at[0];
        k = s_at[1];
        if (!s_at[2]) break;
    }
    if (t < 32) {
        if (v > 0 && h > 0) {
            const int run = min(v, h);
            pos = emit_run_g<32>(slot, pos, run, 'M', 'M', lane, A.err);
            v -= run;
            h -= run;
        }
        pos = emit_run_g<32>(slot, pos, v, 'D', 'D', lane, A.err);
        pos = emit_run_g<32>(slot, pos, h, 'I', 'I', lane, A.err);
    }
    return pos;
}

template <bool TRACE>
__global__ void __launch_bounds__(BLK_T, 2) wfa_block_kernel(WfaBlockArgs B)
{
    extern __shared__ __align__(16) int32_t bsmem[];
    __shared__ int s_q, s_at[3];
    const WfaArgs& A = B.A;
    const int t = threadIdx.x, smax = A.smax;
    // (the pairs that look longest before the rest of those left)
    const int nbig = B.big_count ? *B.big_count : 0, nfar = nbig + (A.far_count ? *A.far_count : 0);
    const int left = A.blk_count ? *A.blk_count : 0, cnt = nfar + (left > B.few ? 0 : left);
    int32_t* const wf0 = bsmem;
    int32_t* const wf1 = bsmem + 2 * smax + 3;
    int32_t* const stk = TRACE ? A.stack + blockIdx.x * ((int64_t)(smax + 1) * (smax + 1)) : nullptr;
    auto next_item = [&]() {
        if (t == 0) s_q = gridDim.x + atomicAdd(B.next, 1);
        __syncthreads();
        const int q = s_q;
        __syncthreads();
        return q;
    };
    for (int q = first_item(blockIdx.x, gridDim.x, B.packed); q < cnt; q = next_item()) {
        const int p = q < nbig ? B.big[q].x : (q < nfar ? A.far[q - nbig] : A.blk[q - nfar]);
        const int m = A.D.a_len[p], n = A.D.b_len[p];
        if (m <= 0 || n <= 0) {
            const int len = m <= 0 ? max(n, 0) : m;
            const char op = m <= 0 ? 'I' : 'D';
            if (TRACE) emit_run_g<BLK_T>(A.out_cigar + A.D.out_off[p], len, len, op, op, t, A.err);
            if (t == 0) {
                A.out_score[p] = len;
                if (A.out_len) A.out_len[p] = TRACE ? len : 0;
            }
            continue;
        }
        int score;
        if (A.D.pure[p] && A.D.pure[A.D.n + p])
            score = wfa_forward<TRACE, 2, BLK_T>(A.D.packed + (A.D.a_off[p] >> 5), A.D.packed + (A.D.b_off[p] >> 5), m, n,
                                                 smax, wf0, wf1, stk, t, FULL);
        else
            score = wfa_forward<TRACE, 8, BLK_T>(reinterpret_cast<const uint64_t*>(A.D.seq + A.D.a_off[p]),
                                                 reinterpret_cast<const uint64_t*>(A.D.seq + A.D.b_off[p]), m, n, smax,
                                                 wf0, wf1, stk, t, FULL);
        int len = 0;
        if (TRACE && score >= 0) {
            __syncthreads();                       // the wavefronts are read; their memory is the walk's now
            const int pos = score == 0 ? emit_run_g<BLK_T>(A.out_cigar + A.D.out_off[p], m + n, n, 'M', 'M', t, A.err)
                                       : walk_block(A, p, score, n - m, m, n, stk, bsmem, s_at);
            len = m + n - pos;
        }
        if (t == 0) {
            A.out_score[p] = score;
            if (A.out_len) A.out_len[p] = len;
        }
        __syncthreads();
    }
}

static size_t wfa_block_smem(int smax) { return sizeof(int32_t) * std::max<size_t>(2 * (2 * (size_t)smax + 3), BLK_T); }

int wfa_block_slots(int smax, bool trace, int sm_count)
{
    const size_t smem = wfa_block_smem(smax);
    return (trace ? blocks_per_sm((const void*)wfa_block_kernel<true>, BLK_T, smem)
                  : blocks_per_sm((const void*)wfa_block_kernel<false>, BLK_T, smem)) * sm_count;
}

cudaError_t launch_wfa_block(const WfaBlockArgs& B, int blocks, int kernel_id, cudaStream_t st)
{
    const size_t smem = wfa_block_smem(B.A.smax);
    launch_begin(kernel_id, st);
    if (B.A.trace) wfa_block_kernel<true><<<blocks, BLK_T, smem, st>>>(B);
    else wfa_block_kernel<false><<<blocks, BLK_T, smem, st>>>(B);
    launch_end(kernel_id, st);
    return cudaGetLastError();
}

}  // namespace ga
