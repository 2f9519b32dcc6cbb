// wfa.cu -- sequence packing and the WFA edit-distance kernels (sm_103a).
//
// Algorithm: the wavefront recurrence of the reference's wfa_trace_kernel /
// wfa_score_kernel_flat (include/genoaligner/backend/wfa_kernel.hip:119-145,
// 467-592; wfa_score_flat.hip:63-140).  Offsets are text coordinates h,
// v = h - k, the alignment diagonal is n - m; compute-next takes
// max(del, max(ins, mism) + 1) and clips to NULL past either end before
// extending; the walk prefers mismatch on ties, then insertion, then deletion
// (strictly).  These steps are fixed by the result contract -- the scores and
// CIGAR strings must be the reference's -- so they are kept, expressed for a
// warp:
//
//   * one warp per pair, persistent: warps pull pair indices from a counter,
//     so long and short pairs balance across the grid;
//   * the diagonals of wavefront s are spread over the 32 lanes; the previous
//     and current wavefront live in a per-warp shared-memory ping-pong;
//   * extension compares 16 bases per step on the 2-bit arena (XOR +
//     find-first-set); pairs with any byte outside ACGT compare 8 raw bytes
//     per step instead, so byte-equality semantics hold for N, lowercase, etc.;
//   * for CIGARs every wavefront is also written to a per-warp triangular stack
//     in global memory (wavefront s at s*s, 2s+1 entries); the walk then runs
//     warp-uniformly over it and writes the CIGAR back to front into the
//     pair's output slot, runs of matches written by all lanes at once.
#include "wfa_step.cuh"

namespace ga {

// ---------------------------------------------------------------- packing --
// The 2-bit arena: one thread per 32-byte chunk of the byte arena -> one
// 64-bit word (A=0 C=1 G=2 T=3 under ((c>>1)^(c>>2))&3, little-endian).
// Sequences start on 32-byte boundaries, so word index = byte offset / 32 and
// no per-sequence bookkeeping is needed.
__device__ __forceinline__ void fill_words(const Fills& F)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    for (int k = 0; k < F.count; ++k)
        for (int64_t i = t; i < F.n[k]; i += stride) F.p[k][i] = F.v[k];
}

__global__ void __launch_bounds__(256) pack_chunks_kernel(const uint8_t* __restrict__ seq, int64_t nchunks,
                                                          uint64_t* __restrict__ packed, uint32_t* __restrict__ bad,
                                                          const Fills F)
{
    fill_words(F);
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < nchunks; c += (int64_t)gridDim.x * blockDim.x) {
        const uint4* src = reinterpret_cast<const uint4*>(seq + 32 * c);
        const uint4 x0 = __ldg(src), x1 = __ldg(src + 1);
        const uint32_t parts[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
        uint64_t word = 0;
        uint32_t badbits = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t v = parts[q];
            // four codes of one 32-bit part: ((c >> 1) ^ (c >> 2)) & 3 per byte
            const uint32_t codes = ((v >> 1) ^ (v >> 2)) & 0x03030303u;
            const uint32_t packed4 = (codes & 3u) | ((codes >> 6) & 0xcu) | ((codes >> 12) & 0x30u) | ((codes >> 18) & 0xc0u);
            word |= (uint64_t)packed4 << (8 * q);
            // a byte is A, C, G or T iff it equals "ACGT"[its code]
            const uint32_t sel = (codes & 3u) | ((codes >> 4) & 0x30u) | ((codes >> 8) & 0x300u) | ((codes >> 12) & 0x3000u);
            const uint32_t diff = __byte_perm(0x54474341u, 0u, sel) ^ v;
            const uint32_t nz = ((((diff & 0x7f7f7f7fu) + 0x7f7f7f7fu) | diff) >> 7) & 0x01010101u;
            badbits |= ((nz * 0x10204080u) >> 28) << (4 * q);       // bit 8q+b of nz -> bit 4q+b
        }
        packed[c] = word;
        bad[c] = badbits;
    }
}

// Purity flag per sequence (a-sides q < n, then b-sides) from the per-chunk
// masks of pack_chunks_kernel: bit b of bad[c] = byte 32c + b is not A/C/G/T.
__global__ void __launch_bounds__(256) purity_mask_kernel(PairDesc D, const uint32_t* __restrict__ bad,
                                                          uint8_t* __restrict__ pure)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 2 * D.n; q += gridDim.x * blockDim.x) {
        const bool is_a = q < D.n;
        const int p = is_a ? q : q - D.n;
        const int64_t c0 = (is_a ? D.a_off[p] : D.b_off[p]) >> 5;
        const int len = is_a ? D.a_len[p] : D.b_len[p];
        const int full = len >> 5, rest = len & 31;
        uint32_t acc = 0;
        for (int w = 0; w < full; ++w) acc |= __ldg(bad + c0 + w);
        if (rest) acc |= __ldg(bad + c0 + full) & ((1u << rest) - 1u);
        pure[q] = (uint8_t)(acc == 0);
    }
}

// Letters of each sequence straight from the bytes (the Smith-Waterman paths,
// which build no 2-bit arena): 1 every byte is A, C, G or T; 2 some are N; 0
// some are neither.  G lanes per sequence (purity_lanes), 16 G bytes a step: the
// loads of a sequence are contiguous, and with a warp it takes length / 512 steps
// where a thread takes length / 16 (600 pairs up to 1 kb: 31 -> 7.5 us; 200,000
// uneven pairs, 260 MB: 226 -> 154 us, bound by the latency of the few loads a
// warp has in flight).
template <int G>
__global__ void __launch_bounds__(256) purity_kernel(PairDesc D, uint8_t* __restrict__ pure, const Fills F)
{
    fill_words(F);
    const int lane = threadIdx.x & (G - 1);
    const unsigned gmask = (0xffffffffu >> (32 - G)) << (threadIdx.x & 31 & ~(G - 1));
    const int ng = gridDim.x * blockDim.x / G;
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) / G; q < 2 * D.n; q += ng) {
        const bool is_a = q < D.n;
        const int p = is_a ? q : q - D.n;
        const uint8_t* s = D.seq + (is_a ? D.a_off[p] : D.b_off[p]);
        const int len = is_a ? D.a_len[p] : D.b_len[p];
        uint32_t other = 0, n_seen = 0;                 // bits 0, 8, 16, 24: a byte outside ACGT; an N
        for (int o = 16 * lane; o < len; o += 16 * G) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(s + o));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int left = len - o - 4 * k;       // bytes of this word inside the sequence
                if (left <= 0) break;
                const uint32_t in = left >= 4 ? 0x01010101u : 0x01010101u >> (8 * (4 - left));
                // a byte is A, C, G or T iff it equals "ACGT"[its code]
                const uint32_t codes = ((w[k] >> 1) ^ (w[k] >> 2)) & 0x03030303u;
                const uint32_t sel = (codes & 3u) | ((codes >> 4) & 0x30u) | ((codes >> 8) & 0x300u) | ((codes >> 12) & 0x3000u);
                const uint32_t da = __byte_perm(0x54474341u, 0u, sel) ^ w[k], dn = w[k] ^ 0x4e4e4e4eu;
                const uint32_t not_a = ((((da & 0x7f7f7f7fu) + 0x7f7f7f7fu) | da) >> 7) & in;
                const uint32_t not_n = ((((dn & 0x7f7f7f7fu) + 0x7f7f7f7fu) | dn) >> 7) & in;
                other |= not_a & not_n;
                n_seen |= not_a & ~not_n;
            }
        }
        const bool bad = __any_sync(gmask, other != 0), some_n = __any_sync(gmask, n_seen != 0);
        if (lane == 0) pure[q] = bad ? 0 : (some_n ? 2 : 1);
    }
}

// ------------------------------------------------------------------- WFA --
// Whether a sequence of len bytes whose first chunk's mask is bad[0] is all A, C, G, T.
__device__ __forceinline__ bool side_pure(const uint32_t* __restrict__ bad, int len, int lane)
{
    uint32_t acc = 0;
    for (int w = lane; 32 * w < len; w += 32)
        acc |= __ldg(bad + w) & (len - 32 * w >= 32 ? 0xffffffffu : (1u << (len - 32 * w)) - 1u);
    return !__any_sync(FULL, acc != 0);
}

template <bool TRACE, int BITS, int PASS>
__device__ void wfa_pair(const WfaArgs& A, int p, const uint64_t* __restrict__ P, const uint64_t* __restrict__ T, int m,
                         int n, int32_t* wf0, int32_t* wf1, int32_t* stk, int lane)
{
    const int score = wfa_forward<TRACE, BITS, 32, false, PASS == FIRST_PASS>(P, T, m, n, A.cap, wf0, wf1, stk, lane, FULL);
    if (score < 0 && A.cap < A.smax) {                      // left to another pass or the block kernel
        // past A.far_edits at the rate at which cap edits went through both sides' bases?
        const bool far = PASS == FIRST_PASS && (int64_t)A.cap * (m + n) > (int64_t)A.far_edits * (2 * (-1 - score) - (n - m));
        if (lane == 0) {
            A.pure[p] = A.pure[A.D.n + p] = BITS == 2;
            if (far) A.far[atomicAdd(A.far_count, 1)] = p;
            else A.blk[atomicAdd(A.blk_count, 1)] = p;
        }
        return;
    }
    int len = 0;
    if (TRACE && score >= 0) {
        __syncwarp();                      // stack writes of every lane are visible below
        len = m + n - walk_g<32>(A, p, score, n - m, m, n, stk, lane, FULL);
    }
    if (lane == 0) {
        A.out_score[p] = score;
        if (A.out_len) A.out_len[p] = len;
    }
}

template <bool TRACE, int PASS>
__global__ void __launch_bounds__(128) wfa_kernel(WfaArgs A)
{
    extern __shared__ int32_t smem[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int WS = 2 * A.cap + 3;
    int32_t* wf0 = smem + wib * 2 * WS;
    int32_t* wf1 = wf0 + WS;
    const int64_t slot = (int64_t)blockIdx.x * (blockDim.x >> 5) + wib;
    int32_t* stk = TRACE ? A.stack + slot * A.stack_slot : nullptr;
    const int cnt = PASS == SECOND_PASS ? *A.list_count : A.D.n;
    if (PASS == SECOND_PASS && cnt <= A.list_few) return;    // the block kernel's
    for (;;) {
        int p0 = 0;
        if (lane == 0) p0 = atomicAdd(A.counter, A.chunk);
        p0 = __shfl_sync(FULL, p0, 0);
        if (p0 >= cnt) break;
        const int pend = min(p0 + A.chunk, cnt);
        for (int q = p0; q < pend; ++q) {
        __syncwarp();
        const int p = PASS == SECOND_PASS ? A.list[q] : q;
        const int m = A.D.a_len[p];       // pattern
        const int n = A.D.b_len[p];       // text
        if (m <= 0 || n <= 0) {
            // one side empty: the score is the other length, whatever smax is;
            // the CIGAR is all insertions (empty pattern) or all deletions
            // (wfa_kernel.hip:480-502)
            const int len = m <= 0 ? max(n, 0) : m;
            if (TRACE) emit_run_g<32>(A.out_cigar + A.D.out_off[p], len, len, m <= 0 ? 'I' : 'D',
                                      m <= 0 ? 'I' : 'D', lane, A.err);
            if (lane == 0) {
                A.out_score[p] = len;
                if (A.out_len) A.out_len[p] = TRACE ? len : 0;
            }
            continue;
        }
        // both sides pure ACGT: in small batches read from the chunk masks by the warp, where
        // a kernel for the flags would be one more launch (purity_pass; with the fills and
        // the CIGAR packing in their neighbours' kernels, 48 reads took 60 -> 49 us a call)
        bool pure;
        if (A.masks) {
            pure = side_pure(A.masks + (A.D.a_off[p] >> 5), m, lane) & side_pure(A.masks + (A.D.b_off[p] >> 5), n, lane);
        } else {
            pure = A.D.pure[p] && A.D.pure[A.D.n + p];
        }
        if (pure) {
            const uint64_t* P = A.D.packed + (A.D.a_off[p] >> 5);
            const uint64_t* T = A.D.packed + (A.D.b_off[p] >> 5);
            wfa_pair<TRACE, 2, PASS>(A, p, P, T, m, n, wf0, wf1, stk, lane);
        } else {
            const uint64_t* P = reinterpret_cast<const uint64_t*>(A.D.seq + A.D.a_off[p]);
            const uint64_t* T = reinterpret_cast<const uint64_t*>(A.D.seq + A.D.b_off[p]);
            wfa_pair<TRACE, 8, PASS>(A, p, P, T, m, n, wf0, wf1, stk, lane);
        }
        }
    }
}

// --------------------------------------------------------------- launchers --
// Lanes per sequence of purity_kernel: a warp, unless the batch then has more threads
// than the device and a smaller group still reads its mean sequence in four steps.
static int purity_lanes(int n, int64_t seq_bytes)
{
    const int64_t mean = seq_bytes / (2 * (int64_t)n), threads = (int64_t)device_sms() * 2048;
    int g = 32;
    while (g > 1 && 2 * (int64_t)n * g > threads && 32 * g >= mean) g /= 2;
    return g;
}

cudaError_t launch_pack(const PairDesc& D, int64_t seq_bytes, uint64_t* packed, uint8_t* pure, cudaStream_t st,
                        const Fills& fills)
{
    if (fills.over) return cudaErrorInvalidValue;
    if (D.n <= 0) return cudaSuccess;
    int blocks = (2 * D.n + 255) / 256;
    blocks = std::min(blocks, device_sms() * 32);
    if (packed) {
        // every sequence ends >= 64 bytes before the arena's end, so the whole
        // chunks cover them all and no read passes seq_bytes
        const int64_t nchunks = seq_bytes / 32;
        uint32_t* bad = packed_masks(packed, seq_bytes);
        int64_t cblocks = (nchunks + 255) / 256;
        cblocks = std::min<int64_t>(cblocks, device_sms() * 32);
        launch_begin(K_PACK, st);
        pack_chunks_kernel<<<(int)std::max<int64_t>(cblocks, 1), 256, 0, st>>>(D.seq, nchunks, packed, bad, fills);
        launch_end(K_PACK, st);
        if (!pure) return cudaGetLastError();
        launch_begin(K_PACK, st);
        purity_mask_kernel<<<blocks, 256, 0, st>>>(D, bad, pure);
        launch_end(K_PACK, st);
        return cudaGetLastError();
    }
    launch_begin(K_PACK, st);
    const int g = purity_lanes(D.n, seq_bytes);
    blocks = (int)std::min<int64_t>((2 * (int64_t)D.n * g + 255) / 256, (int64_t)device_sms() * 32);
    auto kernel = g == 32 ? purity_kernel<32> : g == 16 ? purity_kernel<16> : g == 8 ? purity_kernel<8>
                : g == 4  ? purity_kernel<4>  : g == 2  ? purity_kernel<2>  : purity_kernel<1>;
    kernel<<<blocks, 256, 0, st>>>(D, pure, fills);
    launch_end(K_PACK, st);
    return cudaGetLastError();
}

// The 2-bit words and non-ACGT masks of a whole byte arena (seq_bytes a
// multiple of 32, seq 16-byte aligned): packed[c], bad[c] for every chunk c.
cudaError_t launch_pack_arena(const uint8_t* seq, int64_t seq_bytes, uint64_t* packed, uint32_t* bad, cudaStream_t st)
{
    const int64_t nchunks = seq_bytes / 32;
    if (nchunks <= 0) return cudaSuccess;
    int64_t cblocks = (nchunks + 255) / 256;
    cblocks = std::min<int64_t>(cblocks, device_sms() * 32);
    launch_begin(K_PACK, st);
    pack_chunks_kernel<<<(int)cblocks, 256, 0, st>>>(seq, nchunks, packed, bad, Fills());
    launch_end(K_PACK, st);
    return cudaGetLastError();
}

// The result checks of the reference's validate (src/api/api.cpp:84-112), one
// warp per pair over its CIGAR (at the end of its slot), 32 ops at a time:
// each lane's op steps the pattern and/or the text, a warp prefix sum gives
// its position, and the lanes check their M / X bytes together (the ops and
// the bytes they compare are read contiguously).  Wellformed when the ops
// consume exactly the pattern and the text with M only on equal bytes and X
// only on unequal ones; rescore when the X, I and D ops number the score.
// flags[p] = rescore_ok | wellformed_ok << 1 for pairs with a CIGAR, 0 for
// the others.
__global__ void wfa_validate_kernel(PairDesc D, const int32_t* __restrict__ score, const int32_t* __restrict__ len,
                                    const char* __restrict__ cig, uint8_t* __restrict__ flags,
                                    const int64_t* __restrict__ pk_off, uint8_t* __restrict__ pk)
{
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < D.n; p += nw) {
        const int s = score[p], L = len[p];
        if (s < 0 || L <= 0) {                         // no CIGAR: len may hold anything
            if (lane == 0) flags[p] = 0;
            continue;
        }
        uint8_t* dst = pk ? pk + pk_off[p] : nullptr;
        const int m = D.a_len[p], n = D.b_len[p];
        const uint8_t* P = D.seq + D.a_off[p];
        const uint8_t* T = D.seq + D.b_off[p];
        const char* cg = cig + D.out_off[p] + (m + n) - L;
        int pi0 = 0, ti0 = 0, cost = 0;                            // cost: this lane's ops
        // the ops are loaded a step ahead and the bytes of an M or X compared a step
        // behind, so a lone warp waits for neither
        bool bad = false, chk = false, chk_m = false;
        uint8_t cp = 0, ct = 0;
        char next = lane < L ? cg[lane] : 'I';
        for (int q0 = 0; q0 < L; q0 += 32) {
            const int q = q0 + lane;
            const char op = next;
            next = q + 32 < L ? cg[q + 32] : 'I';
            const bool mx = op == 'M' || op == 'X';
            const int dp = (mx || op == 'D') && q < L, dt = (mx || op == 'I') && q < L;
            int v = dp << 16 | dt;                                 // inclusive prefix of both steps
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL, v, o);
                if (lane >= o) v += y;
            }
            const int pi = pi0 + (v >> 16) - dp, ti = ti0 + (v & 0xffff) - dt;
            bad |= chk && (cp == ct) != chk_m;
            chk = false;
            if (q < L) {
                if (mx) {
                    chk = pi < m && ti < n;
                    bad |= !chk;
                    chk_m = op == 'M';
                    if (chk) { cp = P[pi]; ct = T[ti]; }
                } else {
                    bad |= op != 'I' && op != 'D';
                }
                cost += op == 'X' || op == 'I' || op == 'D';
            }
            if (pk) pack_ops(dst, op, q, L, lane);
            const int tot = __shfl_sync(FULL, v, 31);
            pi0 += tot >> 16;
            ti0 += tot & 0xffff;
        }
        bad |= chk && (cp == ct) != chk_m;
        bad = __any_sync(FULL, bad);
        cost = __reduce_add_sync(FULL, cost);
        if (lane == 0) flags[p] = (uint8_t)((cost == s ? 1 : 0) | (!bad && pi0 == m && ti0 == n ? 2 : 0));
    }
}

// A warp per pair, each side's bytes copied 32 at a time (one sector read and
// written per step; the destination is 32-byte aligned).
__global__ void gather_sides_kernel(PairDesc D, uint8_t* __restrict__ seq, const uint8_t* __restrict__ span_a,
                                    const uint8_t* __restrict__ span_b, const int64_t* __restrict__ src_a,
                                    const int64_t* __restrict__ src_b)
{
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < D.n; p += nw) {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int64_t src = side ? src_b[p] : src_a[p];
            if (src < 0) continue;
            const int len = side ? D.b_len[p] : D.a_len[p];
            const uint8_t* s = (side ? span_b : span_a) + src;
            uint8_t* d = seq + (side ? D.b_off[p] : D.a_off[p]);
            for (int k = lane; k < len; k += 32) d[k] = s[k];
        }
    }
}

cudaError_t launch_gather_sides(const PairDesc& D, uint8_t* seq, const uint8_t* span_a, const uint8_t* span_b,
                                const int64_t* src_a, const int64_t* src_b, cudaStream_t st)
{
    if (D.n <= 0) return cudaSuccess;
    const int blocks = (int)std::min<int64_t>(((int64_t)D.n + 3) / 4, (int64_t)device_sms() * 16);   // a warp per pair
    launch_begin(K_PACK, st);
    gather_sides_kernel<<<blocks, 128, 0, st>>>(D, seq, span_a, span_b, src_a, src_b);
    launch_end(K_PACK, st);
    return cudaGetLastError();
}

cudaError_t launch_wfa_validate(const PairDesc& D, const int32_t* score, const int32_t* len, const char* cig,
                                uint8_t* flags, cudaStream_t st, const int64_t* pk_off, uint8_t* pk)
{
    if (D.n <= 0) return cudaSuccess;
    const int blocks = (int)std::min<int64_t>(((int64_t)D.n + 3) / 4, (int64_t)device_sms() * 16);   // a warp per pair
    launch_begin(K_VALIDATE, st);
    wfa_validate_kernel<<<blocks, 128, 0, st>>>(D, score, len, cig, flags, pk_off, pk);
    launch_end(K_VALIDATE, st);
    return cudaGetLastError();
}

// 64-bit words of a packed arena for seq_bytes of sequence: the 2-bit words
// (+2 spare, read by two-word fetch windows) then one 32-bit mask per chunk.
int64_t packed_arena_words(int64_t seq_bytes)
{
    const int64_t nchunks = seq_bytes / 32;
    return nchunks + 2 + (nchunks + 1) / 2;
}

size_t wfa_smem_bytes(int smax) { return (size_t)4 * 2 * (2 * smax + 3) * sizeof(int32_t); }

using WfaKernel = void (*)(WfaArgs);
static WfaKernel wfa_kernel_of(bool trace, int pass)
{
    if (pass == FIRST_PASS) return trace ? wfa_kernel<true, FIRST_PASS> : wfa_kernel<false, FIRST_PASS>;
    if (pass == SECOND_PASS) return trace ? wfa_kernel<true, SECOND_PASS> : wfa_kernel<false, SECOND_PASS>;
    return trace ? wfa_kernel<true, ONLY_PASS> : wfa_kernel<false, ONLY_PASS>;
}

int wfa_max_slots(int smax, bool trace, int sm_count, int pass)
{
    return blocks_per_sm((const void*)wfa_kernel_of(trace, pass), 128, wfa_smem_bytes(smax)) * sm_count * 4;
}

cudaError_t launch_wfa(const WfaArgs& A, int slots, cudaStream_t st)
{
    if (A.D.n <= 0) return cudaSuccess;
    const int blocks = (slots + 3) / 4;
    const size_t smem = wfa_smem_bytes(A.cap);
    const int id = A.trace ? K_WFA_TRACE : K_WFA_SCORE;
    launch_begin(id, st);
    const WfaKernel kernel = wfa_kernel_of(A.trace, A.list ? SECOND_PASS : (A.far ? FIRST_PASS : ONLY_PASS));
    kernel<<<blocks, 128, smem, st>>>(A);
    launch_end(id, st);
    return cudaGetLastError();
}

}  // namespace ga
