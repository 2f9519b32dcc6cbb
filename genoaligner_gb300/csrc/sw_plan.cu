// sw_plan.cu -- the Smith-Waterman traceback work plan, built on the device.
//
// The plan sorts the pairs of a batch into the kernels' work lists, largest
// first: the two-pairs-per-warp 16-bit list (A, C, G, T, N pairs whose scores fit
// 16 bits; consecutive entries share a warp) and the 32-bit lists (short and
// long shapes of sw32ck.cu).  It is a counting sort on a size key (16-bit
// pairs: forward column extent, then rows; 32-bit pairs: 64 buckets per
// doubling of (m + 31) * n) in four kernels -- classify and
// count, scan, scatter, pack -- or, for a small batch, in one block, and leaves on the device the work lists in
// the order the launches read them plus, per list, its length and the largest
// per-warp memory its items need.  The host entry's launches read that small
// record on the device (plan mode: grids and memory sized from host bounds);
// the device entry reads it back to size its memory exactly.
#include "kernels.cuh"

namespace ga {

constexpr int SP_NB = 4096;              // size buckets per list

// Bucket of a 16-bit pair (sw16_shape_key).
__device__ __forceinline__ int sp_key16(int m, int n) { return sw16_shape_key(m, n); }

// Bucket of a 32-bit pair of m rows and n columns, largest first.
__device__ __forceinline__ int sp_key(int m, int n)
{
    const uint64_t c = (uint64_t)(max(m, 0) + 31) * (uint64_t)max(n, 1);
    const int lz = __clzll((long long)c), e = 63 - lz;
    const int frac = (int)(((c << lz) >> 57) & 63u);
    return SP_NB - 1 - min(SP_NB - 1, e * 64 + frac);
}

// What the pairs of one list, or of one block's share of it, add to the record.
struct SpTally {
    unsigned long long cells[SP_LISTS], largest[SP_LISTS], nopt, diropt, edge;
    int cols[SP_LISTS];
};

// Pair p's bucket, list * SP_NB + key (-1: no list; too large for a trace), its part of
// the record added to the thread's tally.
__device__ __forceinline__ int sp_classify(const SwPlanArgs& P, int p, SpTally& T)
{
    const int n = P.D.n, m = P.D.a_len[p], nn = P.D.b_len[p];
    if (P.cell_limit >= 0 && m > 0 && nn > 0 && ((int64_t)m + 1) * ((int64_t)nn + 1) > P.cell_limit) {
        P.out_score[p] = P.too_large_score;
        return -1;
    }
    const bool pure = P.use16 && P.D.pure[p] && P.D.pure[n + p] && (P.score_only || m <= SW16_TRACE_ROWS);
    const bool strict = pure && sw16_eligible(m, nn, P.match, P.mismatch, P.gap_open, P.gap_extend);
    const bool opt = P.try16 ? (P.try16[p] != 0 && m > 0 && nn > 0 &&
                                sw16_scheme_ok(P.match, P.mismatch, P.gap_open, P.gap_extend))
                             : sw16_eligible_opt(m, nn, P.match, P.mismatch, P.gap_open, P.gap_extend, P.opt16_pct);
    const bool tried = !P.score_only && pure && opt && !strict, u16 = strict || (tried && P.handover);
    if (tried) {                    // may be handed to the 32-bit long-shape kernel
        ++T.nopt;
        T.diropt = max(T.diropt, (unsigned long long)sw32ck_dir_words(m, nn, 0));
    }
    const int list = u16 ? SP_L16 : ((!P.score_only && sw32ck_long(m, nn, P.long_log2)) ? SP_L32LONG : SP_L32);
    T.edge = max(T.edge, (unsigned long long)(2 * max(m, 0)));
    const unsigned long long c = (unsigned long long)max(m, 0) * (unsigned long long)max(nn, 0);
#pragma unroll
    for (int l = 0; l < SP_LISTS; ++l)
        if (l == list) {
            T.cells[l] += c;
            T.largest[l] = max(T.largest[l], c);
            T.cols[l] = max(T.cols[l], nn);
        }
    return list * SP_NB + (u16 ? sp_key16(m, nn) : sp_key(m, nn));
}

__device__ __forceinline__ unsigned long long sp_max(unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

// A warp's tallies into a record (in shared or global memory).
__device__ __forceinline__ void sp_add_tally(const SpTally& T, unsigned long long* res, int lane)
{
#pragma unroll
    for (int l = 0; l < SP_LISTS; ++l) {
        unsigned long long c = T.cells[l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
        const unsigned long long g = sp_max(T.largest[l]);
        const int cols = __reduce_max_sync(FULL, T.cols[l]);
        if (lane == 0 && g) {
            atomicAdd(res + SP_CELLS + l, c);
            atomicMax(res + SP_LARGEST + l, g);
            atomicMax(res + SP_COLS + l, (unsigned long long)cols);
        }
    }
    const unsigned nopt = __reduce_add_sync(FULL, (unsigned)T.nopt);
    const unsigned long long diropt = sp_max(T.diropt), edge = sp_max(T.edge);
    if (lane == 0) {
        if (nopt) {
            atomicAdd(res + SP_NOPT, (unsigned long long)nopt);
            atomicMax(res + SP_DIROPT, diropt);
        }
        if (edge) atomicMax(res + SP_EDGE, edge);
    }
}

__global__ void sp_classify_kernel(SwPlanArgs P)
{
    __shared__ unsigned long long rec[SP_RES];
    const int lane = threadIdx.x & 31;
    const int n = P.D.n;
    const int stride = gridDim.x * blockDim.x;
    if (threadIdx.x < SP_RES) rec[threadIdx.x] = 0;
    __syncthreads();
    SpTally T{};
    for (int p0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); p0 < n; p0 += stride) {
        const int p = p0 + lane;
        const int it = p < n ? sp_classify(P, p, T) : -1;
        if (p < n) P.item[p] = it;
        const unsigned same = __match_any_sync(FULL, it);
        if (it >= 0 && lane == __ffs(same) - 1) atomicAdd(&P.counts[it], __popc(same));
    }
    sp_add_tally(T, rec, lane);
    __syncthreads();
    const int k = threadIdx.x;
    if (k < SP_RES && rec[k]) {
        unsigned long long* r = reinterpret_cast<unsigned long long*>(P.res) + k;
        if (k == SP_NOPT || (k >= SP_CELLS && k < SP_CELLS + SP_LISTS)) atomicAdd(r, rec[k]);
        else atomicMax(r, rec[k]);
    }
}

// Cells that the list's items cost the device's warps: an item of the 16-bit list holds
// two pairs and costs a warp what one does, and the ranges beside this one cost the same.
__device__ __forceinline__ int64_t sp_item_cells(const SwPlanArgs& P, const long long* res, int l)
{
    return (int64_t)P.parts * (l == SP_L16 ? res[SP_CELLS + l] / 2 : res[SP_CELLS + l]);
}

// Lists' lengths in the flattened work array and their offsets there (16-bit lists
// hold two entries per work item), the warps of their whole-block launches, and
// whether the launches that follow serve these lists.
__device__ __forceinline__ void sp_lay_out(const SwPlanArgs& P, long long* res, const long long* total)
{
    long long base = 0;
    bool served = res[SP_NOPT] == 0 || P.handover;
    for (int l = 0; l < SP_LISTS; ++l) {
        const long long ints = l == SP_L16 ? 2 * ((total[l] + 1) / 2) : total[l];
        served = served && (total[l] == 0 || (P.launched >> l & 1));
        res[SP_COUNT + l] = total[l];
        res[SP_INTS + l] = ints;
        res[SP_BASE + l] = base;
        base += ints;
        res[SP_COOPW + l] = P.coop_block[l] ? P.coop_block[l]
                                            : sw_coop_block(res[SP_LARGEST + l], (int)res[SP_COLS + l],
                                                            sp_item_cells(P, res, l), P.sms);
    }
    if (!served && P.err) atomicOr(P.err, ERR_SCRATCH);
}

// Work items first, first + step, ... of list l in launch order; their largest
// per-warp memory, and the list's leading whole-block items: those up to the last item
// above sp_coop_cells.  The 32-bit lists come by cells, the 16-bit list only among its
// widest pairs, so there only those count, unless the items are so few that each can
// have a block.
__device__ __forceinline__ void sp_pack_list(const SwPlanArgs& P, const long long* res, int l, const int32_t* srt,
                                             long long first, long long step, unsigned long long& local,
                                             unsigned long long& ncoop)
{
    const long long cnt = res[SP_COUNT + l];
    int32_t* w = P.work + res[SP_BASE + l];
    const int64_t cells = sp_item_cells(P, res, l), all = P.parts * (l == SP_L16 ? (cnt + 1) / 2 : cnt);
    const bool even = P.decide_even && sw_even_many(all, res[SP_LARGEST + l], cells, (int)res[SP_COLS + l], P.coop_warps[l]);
    const int64_t coop = even ? INT64_MAX : sp_coop_cells(P.coop_limit, cells, P.coop_warps[l]);
    const int W = (int)res[SP_COOPW + l];
    if (l == SP_L16) {
        const long long items = (cnt + 1) / 2;
        const bool few = W * items * P.parts <= P.coop_warps[l];
        for (long long q = first; q < items; q += step) {
            const int a = srt[2 * q], b = 2 * q + 1 < cnt ? srt[2 * q + 1] : -1;
            w[2 * q] = a;
            w[2 * q + 1] = b;
            const int M = max(P.D.a_len[a], b >= 0 ? P.D.a_len[b] : 0);
            const int N = max(P.D.b_len[a], b >= 0 ? P.D.b_len[b] : 0);
            int64_t words = P.score_only ? sw16so_dir_words(M, N) : sw16ck_dir_words(M, N, P.window);
            if ((int64_t)M * N > coop && (few || sw16_by_cells(N))) {
                ncoop = q + 1;
                words = sw_coop_share(words, W, sw16_own_words(!P.score_only, P.window));
            }
            local = max(local, (unsigned long long)words);
        }
        return;
    }
    for (long long q = first; q < cnt; q += step) {
        const int a = srt[q];
        w[q] = a;
        if (P.score_only) continue;
        int64_t words = sw32ck_dir_words(P.D.a_len[a], P.D.b_len[a], P.long_log2);
        if ((int64_t)P.D.a_len[a] * P.D.b_len[a] > coop) {
            ncoop = q + 1;
            words = sw_coop_share(words, W, sw32_own_words(P.D.a_len[a], P.D.b_len[a], P.long_log2));
        }
        local = max(local, (unsigned long long)words);
    }
}

// Exclusive scan of each list's bucket counts (bucket order is largest first) by one
// block of NT threads: start[l][b] for list l's bucket b, in cnt's place or in
// another array (flat: counted on from list to list); the lists' totals.
template <int NT>
__device__ __forceinline__ void sp_scan(const int32_t* cnt, int32_t* start, bool flat, int32_t (*warp_sum)[32],
                                        long long* total)
{
    constexpr int BPT = SP_NB / NT;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int own[SP_LISTS], incl[SP_LISTS];
#pragma unroll
    for (int l = 0; l < SP_LISTS; ++l) {
        own[l] = 0;
#pragma unroll
        for (int k = 0; k < BPT; ++k) own[l] += cnt[l * SP_NB + tid * BPT + k];
        incl[l] = own[l];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl[l], o);
            if (lane >= o) incl[l] += v;
        }
        if (lane == 31) warp_sum[l][wid] = incl[l];
    }
    __syncthreads();
    if (wid < SP_LISTS) {
        const int v = lane < NT / 32 ? warp_sum[wid][lane] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(FULL, s, o);
            if (lane >= o) s += u;
        }
        warp_sum[wid][lane] = s - v;
        if (lane == 31) total[wid] = s;
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < SP_LISTS; ++l) {
        int acc = warp_sum[l][wid] + incl[l] - own[l];
        if (flat)                                      // one array for all lists: behind the lists before
            for (int k = 0; k < l; ++k) acc += (int)total[k];
#pragma unroll
        for (int k = 0; k < BPT; ++k) {
            const int c = cnt[l * SP_NB + tid * BPT + k];
            start[l * SP_NB + tid * BPT + k] = acc;
            acc += c;
        }
    }
}

// (A warp per list, 128 buckets a lane, took 30 us of a 200,000-pair plan; 1,024
// threads 7.)
template <int NT>
__global__ void __launch_bounds__(NT) sp_scan_kernel(SwPlanArgs P)
{
    __shared__ long long total[SP_LISTS];
    __shared__ int32_t warp_sum[SP_LISTS][32];
    sp_scan<NT>(P.counts, P.starts, false, warp_sum, total);
    if (threadIdx.x == 0) sp_lay_out(P, P.res, total);
}

__global__ void sp_scatter_kernel(SwPlanArgs P)
{
    const int lane = threadIdx.x & 31;
    const int n = P.D.n;
    const int stride = gridDim.x * blockDim.x;
    for (int p0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); p0 < n; p0 += stride) {
        const int p = p0 + lane;
        const int it = p < n ? P.item[p] : -1;
        const unsigned same = __match_any_sync(FULL, it);
        const int leader = __ffs(same) - 1;
        int base = 0;
        if (it >= 0 && lane == leader) base = atomicAdd(&P.starts[it], __popc(same));
        base = __shfl_sync(FULL, base, leader);
        if (it >= 0) P.sorted[(int64_t)(it / SP_NB) * n + base + __popc(same & ((1u << lane) - 1u))] = p;
    }
}

__global__ void sp_pack_kernel(SwPlanArgs P)
{
    for (int l = 0; l < SP_LISTS; ++l) {
        if (P.res[SP_COUNT + l] == 0) continue;
        unsigned long long local = 0, ncoop = 0;
        sp_pack_list(P, P.res, l, P.sorted + (int64_t)l * P.D.n, blockIdx.x * blockDim.x + threadIdx.x,
                     gridDim.x * blockDim.x, local, ncoop);
        local = sp_max(local);
        ncoop = sp_max(ncoop);
        unsigned long long* r = reinterpret_cast<unsigned long long*>(P.res) + l;
        if ((threadIdx.x & 31) == 0 && local) atomicMax(r + SP_DIR, local);
        if ((threadIdx.x & 31) == 0 && ncoop) atomicMax(r + SP_NCOOP, ncoop);
    }
}

// The same plan by one block, for at most SP_SMALL pairs: the four kernels' launches
// and the trips through memory between them cost a small batch more than the work
// (plan of one pair 51 -> 11 us; a call of 4,096 pairs 399 us either way, of 8,192 pairs
// 558 us by one block and 541 by four kernels, of 16,384 pairs 933 and 886).  A
// pair's place in its bucket is what its count's atomic returns.
constexpr int SP_SMALL = 4096, SP_SMALL_T = 1024;
__global__ void __launch_bounds__(SP_SMALL_T) sp_small_kernel(SwPlanArgs P)
{
    extern __shared__ int32_t sp_smem[];
    int32_t* cnt = sp_smem;                            // SP_LISTS x SP_NB
    int32_t* sorted = sp_smem + SP_LISTS * SP_NB;      // SP_SMALL, list after list
    __shared__ unsigned long long rec[SP_RES];
    __shared__ int32_t warp_sum[SP_LISTS][32];
    __shared__ long long total[SP_LISTS];
    const int n = P.D.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int PER = SP_SMALL / SP_SMALL_T;
    for (int k = tid; k < SP_LISTS * SP_NB; k += SP_SMALL_T) cnt[k] = 0;
    if (tid < SP_RES) rec[tid] = 0;
    __syncthreads();
    SpTally T{};
    int it[PER], at[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int p = tid + k * SP_SMALL_T;
        it[k] = p < n ? sp_classify(P, p, T) : -1;
        at[k] = it[k] >= 0 ? atomicAdd(&cnt[it[k]], 1) : 0;
    }
    if (wid * 32 < n) sp_add_tally(T, rec, lane);
    __syncthreads();
    sp_scan<SP_SMALL_T>(cnt, cnt, true, warp_sum, total);
    if (tid == 0) sp_lay_out(P, reinterpret_cast<long long*>(rec), total);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k)
        if (it[k] >= 0) sorted[cnt[it[k]] + at[k]] = tid + k * SP_SMALL_T;
    __syncthreads();
    int first = 0;
    for (int l = 0; l < SP_LISTS; ++l) {
        if (total[l] > 0) {
            unsigned long long local = 0, ncoop = 0;
            sp_pack_list(P, reinterpret_cast<const long long*>(rec), l, sorted + first, tid, SP_SMALL_T, local, ncoop);
            local = sp_max(local);
            ncoop = sp_max(ncoop);
            if (lane == 0 && local) atomicMax(&rec[SP_DIR + l], local);
            if (lane == 0 && ncoop) atomicMax(&rec[SP_NCOOP + l], ncoop);
        }
        first += (int)total[l];
    }
    __syncthreads();
    if (tid < SP_RES) P.res[tid] = (long long)rec[tid];
}

// ------------------------------------------------------------ validation --
// The result checks of the reference's sw_validate (src/api/api.cpp:114-156),
// one warp per pair over its CIGAR (written at the end of its slot), 32 ops at
// a time: each lane's op steps the text and/or the pattern, a warp prefix sum
// gives its cell, and the lanes check their ops together.  The ops must
// consume exactly the span [start, end] of both sequences, M only on equal
// bytes and X on unequal ones (wellformed), and re-score to the reported
// score (rescore), each gap run costing gap_open + (L - 1) * gap_extend:
// L * gap_extend per gap op plus gap_open - gap_extend per run, a run
// starting at an I (or D) whose previous op is not one.  flags[p] =
// rescore_ok | wellformed_ok << 1 for pairs with a CIGAR, 0 otherwise.
__global__ void sw_validate_kernel(PairDesc D, int match, int mismatch, int go, int ge, const int32_t* __restrict__ score,
                                   const int32_t* __restrict__ pos, const int32_t* __restrict__ len,
                                   const char* __restrict__ cig, uint8_t* __restrict__ flags,
                                   const int64_t* __restrict__ pk_off, uint8_t* __restrict__ pk)
{
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < D.n; p += nw) {
        const int s = score[p], L = len[p];
        if (s <= 0 || L <= 0) {                        // no CIGAR: len and pos may hold anything
            if (lane == 0) flags[p] = 0;
            continue;
        }
        uint8_t* dst = pk ? pk + pk_off[p] : nullptr;
        const int m = D.a_len[p], n = D.b_len[p];
        const uint8_t* T = D.seq + D.a_off[p];
        const uint8_t* P = D.seq + D.b_off[p];
        const char* cg = cig + D.out_off[p] + (m + n) - L;
        const int si = pos[4 * p], sj = pos[4 * p + 1], ei = pos[4 * p + 2], ej = pos[4 * p + 3];
        int i0 = si, j0 = sj, total = 0;                            // total: this lane's ops
        // the ops are loaded a step ahead and the bytes of an M or X compared a step
        // behind, so a lone warp waits for neither
        bool bad = false, chk = false, chk_m = false;
        uint8_t ct = 0, cp = 0;
        char prev_last = 0;                                        // the previous chunk's last op
        char next = lane < L ? cg[lane] : 0;
        for (int q0 = 0; q0 < L; q0 += 32) {
            const int q = q0 + lane;
            const bool in = q < L;
            const char op = next;
            next = q + 32 < L ? cg[q + 32] : 0;
            const bool mx = op == 'M' || op == 'X';
            const int di = mx || op == 'I', dj = mx || op == 'D';
            int v = di << 16 | dj;                                 // inclusive prefix of both steps
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL, v, o);
                if (lane >= o) v += y;
            }
            const int i = i0 + (v >> 16) - di, j = j0 + (v & 0xffff) - dj;
            char prev = __shfl_up_sync(FULL, op, 1);
            if (lane == 0) prev = prev_last;
            bad |= chk && (ct == cp) != chk_m;
            chk = false;
            if (in) {
                if (mx) {
                    chk = i <= ei && j <= ej && i < m && j < n;
                    bad |= !chk;
                    chk_m = op == 'M';
                    if (chk) { ct = T[i]; cp = P[j]; }
                    total += op == 'M' ? match : mismatch;
                } else if (op == 'I') {
                    bad |= i > ei || i >= m;
                    total -= ge + (prev != 'I' ? go - ge : 0);
                } else if (op == 'D') {
                    bad |= j > ej || j >= n;
                    total -= ge + (prev != 'D' ? go - ge : 0);
                } else {
                    bad = true;
                }
            }
            if (pk) pack_ops(dst, op, q, L, lane);
            const int tot = __shfl_sync(FULL, v, 31);
            i0 += tot >> 16;
            j0 += tot & 0xffff;
            prev_last = __shfl_sync(FULL, op, 31);
        }
        bad |= chk && (ct == cp) != chk_m;
        total = __reduce_add_sync(FULL, total);
        const bool ok = !__any_sync(FULL, bad) && i0 == ei + 1 && j0 == ej + 1;
        if (lane == 0) flags[p] = (uint8_t)((ok && total == s ? 1 : 0) | (ok ? 2 : 0));
    }
}

cudaError_t launch_sw_validate(const PairDesc& D, const ga_sw_scoring_t& sc, const int32_t* score, const int32_t* pos,
                               const int32_t* len, const char* cig, uint8_t* flags, cudaStream_t st,
                               const int64_t* pk_off, uint8_t* pk)
{
    if (D.n <= 0) return cudaSuccess;
    const int blocks = (int)std::min<int64_t>(((int64_t)D.n + 3) / 4, (int64_t)device_sms() * 16);   // a warp per pair
    launch_begin(K_VALIDATE, st);
    sw_validate_kernel<<<blocks, 128, 0, st>>>(D, sc.match, sc.mismatch, sc.gap_open, sc.gap_extend, score, pos, len,
                                               cig, flags, pk_off, pk);
    launch_end(K_VALIDATE, st);
    return cudaGetLastError();
}

int64_t sw_plan_scratch_ints(int n) { return (int64_t)n + 2 * SP_LISTS * SP_NB + (int64_t)SP_LISTS * n; }

constexpr size_t SP_SMALL_SMEM = sizeof(int32_t) * (SP_LISTS * SP_NB + SP_SMALL);

void sw_plan_prepare() { blocks_per_sm((const void*)sp_small_kernel, SP_SMALL_T, SP_SMALL_SMEM); }

// A range that runs beside others plans while their persistent kernels hold three
// blocks of 128 threads a multiprocessor and 48 of its 64 K registers: a block of 1,024
// threads finds no room there before one of them ends (5 ranges of 4,000 pairs: 170 us
// a launch of four, 520 for the one block), so its plan is made of blocks of 256.
static bool sp_one_block(int n, int parts) { return n <= SP_SMALL && parts == 1; }

void sw_plan_fills(Fills& F, int n, int parts, int32_t* scratch, long long* res)
{
    if (sp_one_block(n, parts)) return;                // sp_small_kernel keeps its own
    F.add(scratch + n, SP_LISTS * SP_NB, 0);           // the buckets' counts
    F.add(res, 2 * SP_RES, 0);
}

cudaError_t launch_sw_plan(SwPlanArgs P, int32_t* scratch, cudaStream_t st)
{
    const int n = P.D.n;
    P.item = scratch;
    P.counts = scratch + n;
    P.starts = P.counts + SP_LISTS * SP_NB;
    P.sorted = P.starts + SP_LISTS * SP_NB;
    if (n <= 0) return cudaSuccess;
    if (sp_one_block(n, P.parts)) {
        launch_begin(K_SWPLAN, st);
        sp_small_kernel<<<1, SP_SMALL_T, SP_SMALL_SMEM, st>>>(P);
        launch_end(K_SWPLAN, st);
        return cudaGetLastError();
    }
    int blocks = (n + 255) / 256;
    blocks = std::min(blocks, device_sms() * 8);
    launch_begin(K_SWPLAN, st);
    sp_classify_kernel<<<blocks, 256, 0, st>>>(P);
    launch_end(K_SWPLAN, st);
    launch_begin(K_SWPLAN, st);
    if (P.parts > 1) sp_scan_kernel<256><<<1, 256, 0, st>>>(P);
    else sp_scan_kernel<1024><<<1, 1024, 0, st>>>(P);
    launch_end(K_SWPLAN, st);
    launch_begin(K_SWPLAN, st);
    sp_scatter_kernel<<<blocks, 256, 0, st>>>(P);
    launch_end(K_SWPLAN, st);
    launch_begin(K_SWPLAN, st);
    sp_pack_kernel<<<blocks, 256, 0, st>>>(P);
    launch_end(K_SWPLAN, st);
    return cudaGetLastError();
}

}  // namespace ga
