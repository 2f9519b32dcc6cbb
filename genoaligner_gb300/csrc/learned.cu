// learned.cu -- the learned cost model: k-mer sketch, MLP forward/backward,
// Adam, all hand-written kernels.
//
// Features of one pair (66 floats): for each of the 64 DNA 3-mers, (count in
// a - count in b) / 8, then len(a) / 256 and len(b) / 256.  3-mers are taken
// on the 2-bit codes ((c >> 1) ^ (c >> 2)) & 3 of the raw bytes, so A/C/G/T
// map to 0..3 and any other byte aliases onto one of them.
//
// The sketch also yields an exact lower bound on the edit distance: an edit
// changes at most 3 3-mers of each string, so d >= L1(count difference) / 6,
// and d >= |len(a) - len(b)|.  Aliasing only merges characters, which can only
// lower the distance of the aliased strings, so the bound holds for the
// original strings.  A pair whose bound exceeds the batch smax is unresolved
// without running WFA -- the same answer the full search gives.
//
// MLP: 66 -> 128 (ReLU) -> 128 (ReLU) -> 2, weights stored as bf16 and
// computed in fp32 (fp32 master copy for Adam).  Outputs: log2(d + 1) and
// log2(wavefront cells + 1) with wavefront cells = (d + 1)^2.  It is a tiny
// GEMM (25k multiply-adds per pair); training runs it as register-tiled fp32 FMA.
#include <atomic>
#include <mutex>
#include <vector>

#include "../../include/genoaligner_gb300.h"
#include "kernels.cuh"
#include "route.cuh"
#include <cuda_bf16.h>

namespace ga {

constexpr int NF = 66, NH1 = 128, NH2 = 128, NO = 2;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH1 * NF, OFF_W2 = OFF_B1 + NH1, OFF_B2 = OFF_W2 + NH2 * NH1,
              OFF_W3 = OFF_B2 + NH2, OFF_B3 = OFF_W3 + NO * NH2, NPARAM = OFF_B3 + NO;

cudaError_t prepare_mlp();
const __nv_bfloat16* cost_model_weights();

// ------------------------------------------------------------------ sketch --
// One warp per pair: 3-mer histograms of both sides in shared memory.
__global__ void __launch_bounds__(256) sketch_kernel(PairDesc D, float* __restrict__ feat,
                                                     int32_t* __restrict__ lower_bound, float s_diff, float s_len)
{
    __shared__ int hist[8][64];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < D.n; p += nwarps) {
        hist[wib][lane] = 0;
        hist[wib][lane + 32] = 0;
        __syncwarp();
        for (int side = 0; side < 2; ++side) {
            const uint8_t* s = D.seq + (side ? D.b_off[p] : D.a_off[p]);
            const int L = side ? D.b_len[p] : D.a_len[p];
            const int sign = side ? -1 : 1;
            for (int q = lane; q + 2 < L; q += 32) {
                const uint32_t c0 = __ldg(s + q), c1 = __ldg(s + q + 1), c2 = __ldg(s + q + 2);
                const int k = (int)((((c0 >> 1) ^ (c0 >> 2)) & 3u) * 16 + (((c1 >> 1) ^ (c1 >> 2)) & 3u) * 4 +
                                    (((c2 >> 1) ^ (c2 >> 2)) & 3u));
                atomicAdd(&hist[wib][k], sign);
            }
        }
        __syncwarp();
        const int d0 = hist[wib][lane], d1 = hist[wib][lane + 32];
        feat[(int64_t)p * NF + lane] = d0 * s_diff;
        feat[(int64_t)p * NF + lane + 32] = d1 * s_diff;
        int l1 = abs(d0) + abs(d1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(FULL, l1, o);
        if (lane == 0) {
            const int m = D.a_len[p], n = D.b_len[p];
            feat[(int64_t)p * NF + 64] = m * s_len;
            feat[(int64_t)p * NF + 65] = n * s_len;
            if (lower_bound) lower_bound[p] = max(abs(m - n), (l1 + 5) / 6);
        }
        __syncwarp();
    }
}

// The same sketch from the 2-bit arena (D.packed).  Lanes 0-15 take side a,
// lanes 16-31 side b; a lane counts the 16 3-mers starting in its 16-base
// stretch from one 64-bit window (3-mer i is bits [2i, 2i+6) of the window).
// The histogram is indexed by the window's own order, c0 + 4 c1 + 16 c2; the
// feature order 16 c0 + 4 c1 + c2 is applied when the features are written.
__global__ void __launch_bounds__(256) sketch_packed_kernel(PairDesc D, float* __restrict__ feat,
                                                            int32_t* __restrict__ lower_bound, float s_diff,
                                                            float s_len)
{
    __shared__ int hist[8][64];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int side = lane >> 4, sl = lane & 15;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < D.n; p += nwarps) {
        hist[wib][lane] = 0;
        hist[wib][lane + 32] = 0;
        __syncwarp();
        const uint64_t* P = D.packed + ((side ? D.b_off[p] : D.a_off[p]) >> 5);
        const int L = side ? D.b_len[p] : D.a_len[p];
        const int sign = side ? -1 : 1;
        for (int q = 16 * sl; q + 2 < L; q += 256) {
            const uint64_t v = fetch_syms<2>(P, q);
            const int cnt = min(16, L - 2 - q);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < cnt) atomicAdd(&hist[wib][(int)((v >> (2 * i)) & 63u)], sign);
        }
        __syncwarp();
        // feature k = 16 c0 + 4 c1 + c2 lives in bin c0 + 4 c1 + 16 c2
        const int k0 = lane, k1 = lane + 32;
        const int d0 = hist[wib][((k0 & 3) << 4) | (k0 & 12) | (k0 >> 4)];
        const int d1 = hist[wib][((k1 & 3) << 4) | (k1 & 12) | (k1 >> 4)];
        feat[(int64_t)p * NF + k0] = d0 * s_diff;
        feat[(int64_t)p * NF + k1] = d1 * s_diff;
        int l1 = abs(d0) + abs(d1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(FULL, l1, o);
        if (lane == 0) {
            const int m = D.a_len[p], n = D.b_len[p];
            feat[(int64_t)p * NF + 64] = m * s_len;
            feat[(int64_t)p * NF + 65] = n * s_len;
            if (lower_bound) lower_bound[p] = max(abs(m - n), (l1 + 5) / 6);
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------- MLP --
// Training and the fp32 forward pass: a block of 512 threads per tile of 64 rows.
// All weights stay in shared memory as fp32 for the block's life (one copy of each
// matrix, [out][in]: a product over `in` reads four of them at once, a product over
// `out` reads rows), and each thread keeps a register tile of its product: 4 x 4 cells
// of a layer, 8 x 4 of dW2, so shared memory is read once per 10 multiply-adds or so
// (twice per multiply-add before).  Bound by FMA issue (66 k multiply-adds a row: the
// products whose operands lie in pairs run two to an instruction) and by the latency
// of eight phases on one tile.  Gradient of 8,192 rows: kernel 150 -> 43.6 us, call
// 182 -> 76 us.  Every sum runs over its index in order, 64 rows to an atomic.  Tiles
// of 16 rows are quicker on batches that leave multiprocessors idle (500 rows: 56 us a
// call against 68), but four times as many atomics carry the sum: relative error 1.0e-7
// against 7.7e-8 there.
constexpr int MLP_T = 512, TILE = 64;
constexpr int MLP_S1 = 68, MLP_S2 = 132;      // row strides: 16-byte rows, 8 rows on 8 bank quads

struct MlpSmem {
    float W1[NH1 * MLP_S1];       // columns 66, 67 zero
    float W2[NH2 * MLP_S2];
    float W3[NO * NH2];
    float b1[NH1], b2[NH2], b3[4];
    float X[TILE * MLP_S1];          // columns 66, 67 zero, rows past the batch zero
    float H1[TILE * MLP_S2];         // then dL/dH1
    float H2[TILE * MLP_S2];         // then dL/dH2
    float y[2 * TILE], dy[2 * TILE], loss[4];
};

__device__ __forceinline__ void load_weights(const __nv_bfloat16* __restrict__ w, MlpSmem& S)
{
    for (int idx = threadIdx.x; idx < NH1 * (NF / 2); idx += MLP_T) {
        const int o = idx / (NF / 2), i = 2 * (idx - o * (NF / 2));
        const float2 v = __bfloat1622float2(*(const __nv_bfloat162*)(w + OFF_W1 + o * NF + i));
        *(float2*)&S.W1[o * MLP_S1 + i] = v;
    }
    for (int o = threadIdx.x; o < NH1; o += MLP_T) *(float2*)&S.W1[o * MLP_S1 + NF] = make_float2(0.f, 0.f);
    for (int idx = threadIdx.x; idx < NH2 * NH1 / 4; idx += MLP_T) {
        const int o = idx / (NH1 / 4), i = 4 * (idx - o * (NH1 / 4));
        const __nv_bfloat162* q = (const __nv_bfloat162*)(w + OFF_W2 + o * NH1 + i);
        const float2 u = __bfloat1622float2(q[0]), v = __bfloat1622float2(q[1]);
        *(float4*)&S.W2[o * MLP_S2 + i] = make_float4(u.x, u.y, v.x, v.y);
    }
    for (int i = threadIdx.x; i < NO * NH2; i += MLP_T) S.W3[i] = __bfloat162float(w[OFF_W3 + i]);
    for (int i = threadIdx.x; i < NH1; i += MLP_T) S.b1[i] = __bfloat162float(w[OFF_B1 + i]);
    for (int i = threadIdx.x; i < NH2; i += MLP_T) S.b2[i] = __bfloat162float(w[OFF_B2 + i]);
    if (threadIdx.x < NO) S.b3[threadIdx.x] = __bfloat162float(w[OFF_B3 + threadIdx.x]);
}

// out[r][o] = max(0, b[o] + sum_i in[r][i] W[o][i]), r < 64, o < 128, i < K.  A warp
// holds 4 row groups x 8 output groups: rows rg + 16 j, outputs cg + 32 k, so both
// operands' 16-byte reads are one shared-memory pass each.
template <int K>
__device__ __forceinline__ void dense_relu(const float* W, int ws, const float* b, const float* in, int is, float* out)
{
    constexpr int NR = TILE / 16;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int rg = (wid & 3) * 4 + (lane >> 3), cg = (wid >> 2) * 8 + (lane & 7);
    float acc[NR][4];
#pragma unroll
    for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[j][k] = b[cg + 32 * k];
#pragma unroll 2
    for (int i = 0; i < K; i += 4) {
        float4 x[NR], v[4];
#pragma unroll
        for (int j = 0; j < NR; ++j) x[j] = *(const float4*)&in[(rg + 16 * j) * is + i];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = *(const float4*)&W[(cg + 32 * k) * ws + i];
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float t = fmaf(x[j].x, v[k].x, acc[j][k]);
                t = fmaf(x[j].y, v[k].y, t);
                t = fmaf(x[j].z, v[k].z, t);
                acc[j][k] = fmaf(x[j].w, v[k].w, t);
            }
    }
#pragma unroll
    for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) out[(rg + 16 * j) * MLP_S2 + cg + 32 * k] = fmaxf(acc[j][k], 0.f);
}

// Rows [base, base + rows) through the network: S.H1, S.H2 and S.y.
__device__ __forceinline__ void forward_tile(const float* __restrict__ feat, int64_t base, int rows, MlpSmem& S)
{
    for (int idx = threadIdx.x; idx < TILE * MLP_S1; idx += MLP_T) {
        const int r = idx / MLP_S1, i = idx - r * MLP_S1;
        S.X[idx] = (r < rows && i < NF) ? feat[(base + r) * NF + i] : 0.f;
    }
    __syncthreads();
    dense_relu<MLP_S1>(S.W1, MLP_S1, S.b1, S.X, MLP_S1, S.H1);
    __syncthreads();
    dense_relu<NH1>(S.W2, MLP_S2, S.b2, S.H1, MLP_S2, S.H2);
    __syncthreads();
    if (threadIdx.x < 2 * TILE) {
        const int r = threadIdx.x >> 1, o = threadIdx.x & 1;
        float acc = S.b3[o];
#pragma unroll 4
        for (int i = 0; i < NH2; i += 4) {
            const float4 h = *(const float4*)&S.H2[r * MLP_S2 + i], v = *(const float4*)&S.W3[o * NH2 + i];
            acc = fmaf(h.x, v.x, acc);
            acc = fmaf(h.y, v.y, acc);
            acc = fmaf(h.z, v.z, acc);
            acc = fmaf(h.w, v.w, acc);
        }
        S.y[threadIdx.x] = acc;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(MLP_T, 1) mlp_forward_kernel(const __nv_bfloat16* __restrict__ w,
                                                            const float* __restrict__ feat, int n, float* __restrict__ y)
{
    extern __shared__ __align__(16) float mlp_smem[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(mlp_smem);
    load_weights(w, S);
    for (int64_t base = (int64_t)blockIdx.x * TILE; base < n; base += (int64_t)gridDim.x * TILE) {
        const int rows = (n - base < TILE) ? (int)(n - base) : TILE;
        forward_tile(feat, base, rows, S);
        for (int idx = threadIdx.x; idx < 2 * rows; idx += MLP_T) y[2 * base + idx] = S.y[idx];
        __syncthreads();
    }
}

__device__ __forceinline__ void add4(float4& a, float s, const float4& v)
{
    const float2 ss = make_float2(s, s);
    const float2 lo = __ffma2_rn(ss, make_float2(v.x, v.y), make_float2(a.x, a.y));
    const float2 hi = __ffma2_rn(ss, make_float2(v.z, v.w), make_float2(a.z, a.w));
    a = make_float4(lo.x, lo.y, hi.x, hi.y);
}

// Forward + backward of the mean squared error over the batch; gradients of
// every parameter (with respect to the bf16-rounded weights) accumulate into
// grad (fp32, 16-byte aligned), the summed squared error behind them.  Blocks add to
// GRAD_COPIES copies in turn and fold_grad_kernel adds the copies: a quarter of the
// partial sums in a row, so a smaller rounding error (8,192 rows: 5.5e-8 relative against
// 1.7e-7 with one copy), for 3 us.
constexpr int GRAD_COPIES = 4, GRAD_STRIDE = (NPARAM + 1 + 3) / 4 * 4;

__global__ void fold_grad_kernel(float* __restrict__ grad)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= NPARAM)
        grad[i] = (grad[i] + grad[GRAD_STRIDE + i]) + (grad[2 * GRAD_STRIDE + i] + grad[3 * GRAD_STRIDE + i]);
}

__global__ void __launch_bounds__(MLP_T, 1) mlp_backward_kernel(const __nv_bfloat16* __restrict__ w,
                                                             const float* __restrict__ feat,
                                                             const float* __restrict__ target, int n,
                                                             float inv_batch, float* __restrict__ grad)
{
    extern __shared__ __align__(16) float mlp_smem[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(mlp_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    grad += (blockIdx.x % GRAD_COPIES) * GRAD_STRIDE;
    load_weights(w, S);
    for (int64_t base = (int64_t)blockIdx.x * TILE; base < n; base += (int64_t)gridDim.x * TILE) {
        const int rows = (n - base < TILE) ? (int)(n - base) : TILE;
        forward_tile(feat, base, rows, S);
        // dL/dy = 2 (y - t) / B
        if (tid < 2 * TILE) {
            float e = 0.f;
            if (tid < 2 * rows) e = S.y[tid] - target[2 * base + tid];
            S.dy[tid] = 2.f * e * inv_batch;
            float lsum = e * e;
            for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(FULL, lsum, o);
            if (lane == 0) S.loss[wid] = lsum;
        }
        __syncthreads();
        // output layer: dW3, db3; dH2 = dy W3 * relu'(H2), H2's column overwritten by the thread that summed it
        if (tid < NH2) {
            const float w0 = S.W3[tid], w1 = S.W3[NH2 + tid];
            float g0 = 0.f, g1 = 0.f, gb = 0.f;
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
                const float2 d = *(const float2*)&S.dy[2 * r];
                float* hp = &S.H2[r * MLP_S2 + tid];
                const float h = *hp;
                g0 = fmaf(d.x, h, g0);
                g1 = fmaf(d.y, h, g1);
                const float g = h > 0.f ? d.x * w0 + d.y * w1 : 0.f;
                gb += g;
                *hp = g;
            }
            atomicAdd(&grad[OFF_W3 + tid], g0);
            atomicAdd(&grad[OFF_W3 + NH2 + tid], g1);
            atomicAdd(&grad[OFF_B2 + tid], gb);
        } else if (tid < NH2 + NO) {
            float g = 0.f;
            for (int r = 0; r < rows; ++r) g += S.dy[2 * r + tid - NH2];
            atomicAdd(&grad[OFF_B3 + tid - NH2], g);
        } else if (tid == NH2 + NO) {
            atomicAdd(&grad[NPARAM], (S.loss[0] + S.loss[1]) + (S.loss[2] + S.loss[3]));
        }
        __syncthreads();
        // layer 2: dW2[o][i] = sum_r dH2[r][o] H1[r][i], 8 outputs (the warp's) x 4 inputs (the lane's) a thread
        {
            float4 acc[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int r = 0; r < rows; ++r) {
                const float4 h = *(const float4*)&S.H1[r * MLP_S2 + 4 * lane];
                const float4 d0 = *(const float4*)&S.H2[r * MLP_S2 + 8 * wid];
                const float4 d1 = *(const float4*)&S.H2[r * MLP_S2 + 8 * wid + 4];
                add4(acc[0], d0.x, h);
                add4(acc[1], d0.y, h);
                add4(acc[2], d0.z, h);
                add4(acc[3], d0.w, h);
                add4(acc[4], d1.x, h);
                add4(acc[5], d1.y, h);
                add4(acc[6], d1.z, h);
                add4(acc[7], d1.w, h);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) atomicAdd((float4*)&grad[OFF_W2 + (8 * wid + k) * NH1 + 4 * lane], acc[k]);
        }
        // dH1[r][i] = sum_o dH2[r][o] W2[o][i] * relu'(H1), in place
        {
            constexpr int NR = TILE / 16;
            const int rg = (wid & 3) * 4 + (lane >> 3), i0 = 4 * ((wid >> 2) * 8 + (lane & 7));
            float4 acc[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int o = 0; o < NH2; o += 4) {
                float4 d[NR], v[4];
#pragma unroll
                for (int j = 0; j < NR; ++j) d[j] = *(const float4*)&S.H2[(rg + 16 * j) * MLP_S2 + o];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = *(const float4*)&S.W2[(o + k) * MLP_S2 + i0];
#pragma unroll
                for (int j = 0; j < NR; ++j) {
                    add4(acc[j], d[j].x, v[0]);
                    add4(acc[j], d[j].y, v[1]);
                    add4(acc[j], d[j].z, v[2]);
                    add4(acc[j], d[j].w, v[3]);
                }
            }
            __syncthreads();                       // dW2 has read H1
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                float4* hp = (float4*)&S.H1[(rg + 16 * j) * MLP_S2 + i0];
                const float4 h = *hp;
                *hp = make_float4(h.x > 0.f ? acc[j].x : 0.f, h.y > 0.f ? acc[j].y : 0.f, h.z > 0.f ? acc[j].z : 0.f,
                                  h.w > 0.f ? acc[j].w : 0.f);
            }
        }
        __syncthreads();
        // layer 1: dW1[o][i] = sum_r dH1[r][o] X[r][i]: 4 x 4 a thread for i < 64, then the last two inputs and db1
        {
            const int o0 = 4 * (tid >> 4), i0 = 4 * (tid & 15);
            float4 acc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            for (int r = 0; r < rows; ++r) {
                const float4 d = *(const float4*)&S.H1[r * MLP_S2 + o0], x = *(const float4*)&S.X[r * MLP_S1 + i0];
                add4(acc[0], d.x, x);
                add4(acc[1], d.y, x);
                add4(acc[2], d.z, x);
                add4(acc[3], d.w, x);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float* g = &grad[OFF_W1 + (o0 + k) * NF + i0];
                atomicAdd((float2*)g, make_float2(acc[k].x, acc[k].y));
                atomicAdd((float2*)(g + 2), make_float2(acc[k].z, acc[k].w));
            }
            if (tid < 2 * NH1) {
                const int o = tid & (NH1 - 1), i = NF - 2 + tid / NH1;
                float g = 0.f;
#pragma unroll 4
                for (int r = 0; r < rows; ++r) g = fmaf(S.H1[r * MLP_S2 + o], S.X[r * MLP_S1 + i], g);
                atomicAdd(&grad[OFF_W1 + o * NF + i], g);
            } else if (tid < 3 * NH1) {
                const int o = tid - 2 * NH1;
                float g = 0.f;
#pragma unroll 4
                for (int r = 0; r < rows; ++r) g += S.H1[r * MLP_S2 + o];
                atomicAdd(&grad[OFF_B1 + o], g);
            }
        }
        __syncthreads();
    }
}

// Adam on the fp32 master copy, then the bf16 copy the forward pass reads.
__global__ void adam_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ w, const float* __restrict__ grad,
                            float* __restrict__ m1, float* __restrict__ m2, int n, float lr, float b1, float b2,
                            float eps, float c1, float c2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float g = grad[i];
        const float a = b1 * m1[i] + (1.f - b1) * g;
        const float v = b2 * m2[i] + (1.f - b2) * g * g;
        m1[i] = a;
        m2[i] = v;
        const float p = master[i] - lr * (a * c1) / (sqrtf(v * c2) + eps);
        master[i] = p;
        w[i] = __float2bfloat16(p);
    }
}

__global__ void to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = __float2bfloat16(src[i]);
}

// ------------------------------------------------- tensor-core inference --
// The routing forward pass on the tensor cores: mma.sync m16n8k16 bf16 with
// fp32 accumulation, one warp per 16 pairs; the inputs and each hidden layer
// are rounded to bf16 as they enter a multiply.  Layer outputs go from the
// accumulator registers straight into the next layer's A fragments (the m16n8
// accumulator layout of two adjacent n-tiles is the A layout of one k16 step).
// Weights are staged once per block in shared memory, rows padded (88 and 136
// bf16) so the eight row groups of a fragment load hit eight bank groups.
constexpr int TK1 = 80, TS1 = 88, TS2 = 136;

struct TcSmem {
    __nv_bfloat16 W1[NH1 * TS1];
    __nv_bfloat16 W2[NH2 * TS2];
    __nv_bfloat16 W3[8 * TS2];
    float b1[NH1], b2[NH2], b3[8];
};

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Weights and biases of a bf16 model into a block's shared memory.
__device__ void load_tc_weights(TcSmem& S, const __nv_bfloat16* __restrict__ w)
{
    for (int idx = threadIdx.x; idx < NH1 * TS1; idx += blockDim.x) {
        const int o = idx / TS1, i = idx - o * TS1;
        S.W1[idx] = i < NF ? w[OFF_W1 + o * NF + i] : __float2bfloat16(0.f);
    }
    for (int idx = threadIdx.x; idx < NH2 * TS2; idx += blockDim.x) {
        const int o = idx / TS2, i = idx - o * TS2;
        S.W2[idx] = i < NH1 ? w[OFF_W2 + o * NH1 + i] : __float2bfloat16(0.f);
    }
    for (int idx = threadIdx.x; idx < 8 * TS2; idx += blockDim.x) {
        const int o = idx / TS2, i = idx - o * TS2;
        S.W3[idx] = (o < NO && i < NH2) ? w[OFF_W3 + o * NH2 + i] : __float2bfloat16(0.f);
    }
    for (int i = threadIdx.x; i < NH1; i += blockDim.x) S.b1[i] = __bfloat162float(w[OFF_B1 + i]);
    for (int i = threadIdx.x; i < NH2; i += blockDim.x) S.b2[i] = __bfloat162float(w[OFF_B2 + i]);
    if (threadIdx.x < 8) S.b3[threadIdx.x] = threadIdx.x < NO ? __bfloat162float(w[OFF_B3 + threadIdx.x]) : 0.f;
}

// One 16-pair tile through the network.  a: the input A fragments (rows g
// and g + 8 of the tile, columns 16 kt + 2 tg (+1, +8, +9)); o: outputs of
// rows g (o[0], o[1]) and g + 8 (o[2], o[3]), valid in lanes with tg == 0.
__device__ __forceinline__ void tc_tile_forward(const TcSmem& S, const uint32_t (&a)[TK1 / 16][4], float (&o)[4])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
    float c[16][4];
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) {
        const float b0 = S.b1[8 * nt + 2 * tg], bb1 = S.b1[8 * nt + 2 * tg + 1];
        c[nt][0] = b0; c[nt][1] = bb1; c[nt][2] = b0; c[nt][3] = bb1;
        const __nv_bfloat16* wr = S.W1 + (8 * nt + g) * TS1 + 2 * tg;
#pragma unroll
        for (int kt = 0; kt < TK1 / 16; ++kt)
            mma_bf16(c[nt], a[kt], *reinterpret_cast<const uint32_t*>(wr + 16 * kt),
                     *reinterpret_cast<const uint32_t*>(wr + 16 * kt + 8));
    }
    uint32_t h[8][4];
#pragma unroll
    for (int kt = 0; kt < 8; ++kt) {
        h[kt][0] = pack_bf16(fmaxf(c[2 * kt][0], 0.f), fmaxf(c[2 * kt][1], 0.f));
        h[kt][1] = pack_bf16(fmaxf(c[2 * kt][2], 0.f), fmaxf(c[2 * kt][3], 0.f));
        h[kt][2] = pack_bf16(fmaxf(c[2 * kt + 1][0], 0.f), fmaxf(c[2 * kt + 1][1], 0.f));
        h[kt][3] = pack_bf16(fmaxf(c[2 * kt + 1][2], 0.f), fmaxf(c[2 * kt + 1][3], 0.f));
    }
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) {
        const float b0 = S.b2[8 * nt + 2 * tg], bb1 = S.b2[8 * nt + 2 * tg + 1];
        c[nt][0] = b0; c[nt][1] = bb1; c[nt][2] = b0; c[nt][3] = bb1;
        const __nv_bfloat16* wr = S.W2 + (8 * nt + g) * TS2 + 2 * tg;
#pragma unroll
        for (int kt = 0; kt < 8; ++kt)
            mma_bf16(c[nt], h[kt], *reinterpret_cast<const uint32_t*>(wr + 16 * kt),
                     *reinterpret_cast<const uint32_t*>(wr + 16 * kt + 8));
    }
#pragma unroll
    for (int kt = 0; kt < 8; ++kt) {
        h[kt][0] = pack_bf16(fmaxf(c[2 * kt][0], 0.f), fmaxf(c[2 * kt][1], 0.f));
        h[kt][1] = pack_bf16(fmaxf(c[2 * kt][2], 0.f), fmaxf(c[2 * kt][3], 0.f));
        h[kt][2] = pack_bf16(fmaxf(c[2 * kt + 1][0], 0.f), fmaxf(c[2 * kt + 1][1], 0.f));
        h[kt][3] = pack_bf16(fmaxf(c[2 * kt + 1][2], 0.f), fmaxf(c[2 * kt + 1][3], 0.f));
    }
    o[0] = S.b3[2 * tg]; o[1] = S.b3[2 * tg + 1]; o[2] = S.b3[2 * tg]; o[3] = S.b3[2 * tg + 1];
    const __nv_bfloat16* wr = S.W3 + g * TS2 + 2 * tg;
#pragma unroll
    for (int kt = 0; kt < 8; ++kt)
        mma_bf16(o, h[kt], *reinterpret_cast<const uint32_t*>(wr + 16 * kt),
                 *reinterpret_cast<const uint32_t*>(wr + 16 * kt + 8));
}

__global__ void __launch_bounds__(256) mlp_forward_tc_kernel(const __nv_bfloat16* __restrict__ w,
                                                             const float* __restrict__ feat, int n,
                                                             float* __restrict__ y)
{
    extern __shared__ __align__(16) unsigned char tc_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(tc_raw);
    load_tc_weights(S, w);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 16 < n; tile += warps) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        auto X = [&](int r, int c) -> float { return (r < n && c < NF) ? __ldg(feat + (int64_t)r * NF + c) : 0.f; };
        uint32_t a[TK1 / 16][4];
#pragma unroll
        for (int kt = 0; kt < TK1 / 16; ++kt) {
            const int c0 = 16 * kt + 2 * tg, c1 = c0 + 8;
            a[kt][0] = pack_bf16(X(r0, c0), X(r0, c0 + 1));
            a[kt][1] = pack_bf16(X(r1, c0), X(r1, c0 + 1));
            a[kt][2] = pack_bf16(X(r0, c1), X(r0, c1 + 1));
            a[kt][3] = pack_bf16(X(r1, c1), X(r1, c1 + 1));
        }
        float o[4];
        tc_tile_forward(S, a, o);
        if (tg == 0) {
            if (r0 < n) { y[2 * (int64_t)r0] = o[0]; y[2 * (int64_t)r0 + 1] = o[1]; }
            if (r1 < n) { y[2 * (int64_t)r1] = o[2]; y[2 * (int64_t)r1 + 1] = o[3]; }
        }
    }
}

// ------------------------------------------ fused routing inference --
// Sketch, lower bound, tensor-core forward pass and queue choice of every pair
// of a WFA batch in one pass, one warp per 16 pairs: lane l < 16 counts the
// 3-mers of side a of pair l of the tile, lane l + 16 those of side b (2^lg lanes a
// side in batches too small for that to use every warp: 16 >> lg pairs), into a
// private histogram column hist[bin][lane] (bin = c0 + 4 c1 + 16 c2, the 2-bit
// window's own order); feature k = 16 c0 + 4 c1 + c2 of pair r is hist[bin][r] -
// hist[bin][r + 16].  Features, bf16 rounding and the network
// are those of ga_wfa_features + ga_mlp_forward_fast, so the prediction is the
// same; nothing but the queue item (route.cuh) leaves the kernel.  MODEL =
// false is the same pass without the network: the queue item comes from the
// exact lower bound alone (the prediction replaced by log2(bound + 1)), for
// measuring what the network adds.
constexpr int RM_WARPS = 16;
constexpr int RM_ROW = 44;        // words of a row of the feature tile: 80 features, rows on distinct banks by fours

template <bool MODEL, bool SPLIT>
__global__ void __launch_bounds__(512) route_model_kernel(const __nv_bfloat16* __restrict__ w, PairDesc D, int smax,
                                                          int lane_smax,
                                                          int32_t* __restrict__ item, int32_t* __restrict__ lb_out,
                                                          float* __restrict__ y_out, int32_t* __restrict__ counts,
                                                          int32_t* __restrict__ out_score, int32_t* __restrict__ out_len,
                                                          int split_log2)
{
    const int lg = SPLIT ? split_log2 : 0;                     // 2^lg lanes to a side: 16 >> lg pairs to a tile
    extern __shared__ __align__(16) unsigned char rm_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(rm_raw);
    int* hist_all = reinterpret_cast<int*>(rm_raw + sizeof(TcSmem));
    __shared__ int local[2 * ROUTE_BUCKETS];
    if (MODEL) load_tc_weights(S, w);
    if (threadIdx.x < 2 * ROUTE_BUCKETS) local[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, g = lane >> 2, tg = lane & 3;
    const int side = lane >> 4, sl = lane & 15;
    int* H = hist_all + wib * 64 * 32 + lane;                 // H[bin * 32]: this lane's column
    const int* Hw = hist_all + wib * 64 * 32;
    const int n = D.n;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * (16 >> lg) < n; tile += warps) {
#pragma unroll 8
        for (int b = 0; b < 64; ++b) H[b * 32] = 0;
        const int p = tile * (16 >> lg) + (sl >> lg);
        int m = 0, nn = 0;
        if (p < n) {
            m = D.a_len[p];
            nn = D.b_len[p];
            const uint64_t* P = D.packed + ((side ? D.b_off[p] : D.a_off[p]) >> 5);
            const int L = side ? nn : m;
            // 256 symbols at a time: the 8 words that hold them and the next
            // one (3-mers straddle it) are loaded together, then counted
            for (int q0 = 256 * (sl & ((1 << lg) - 1)); q0 + 2 < L; q0 += 256 << lg) {
                uint64_t wd[9];
                const int wlast = ((L - 1) >> 5) - (q0 >> 5) + 1;     // words past this lie beyond the arena's spare
#pragma unroll
                for (int j = 0; j < 9; ++j) wd[j] = j <= wlast ? __ldg(P + (q0 >> 5) + j) : 0ull;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int q = q0 + 16 * j;
                    if (q + 2 >= L) break;
                    const uint64_t v = (j & 1) ? ((wd[j >> 1] >> 32) | (wd[(j >> 1) + 1] << 32)) : wd[j >> 1];
                    const int cnt = min(16, L - 2 - q);
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (i < cnt) ++H[(int)((v >> (2 * i)) & 63u) * 32];   // the lane's own column: no atomic
                }
            }
        }
        if (SPLIT && __any_sync(FULL, max(m, nn) > 258)) {
            // a side's lanes each take its counts (with no more than 256 3-mers a side
            // they are its first lane's, the one whose outputs are kept)
#pragma unroll 4
            for (int b = 0; b < 64; ++b) {
                int v = H[b * 32];
                for (int o = 1; o < 1 << lg; o <<= 1) v += __shfl_xor_sync(FULL, v, o);
                H[b * 32] = v;
            }
        }
        __syncwarp();
        // Lanes l and l + 16 take the bins of pair l whose c2 is 0, 1 and 2, 3: each
        // count is read where the bank is the lane's own (its column, then the other
        // side's), the differences give the exact lower bound and, two features to a
        // word, the tile's rows, which then replace the histogram.  (Differences read
        // straight into the fragments met 4-way bank conflicts, the bound's pass 2-way:
        // a third of the pass's shared-memory wavefronts.  1M pairs: 434 -> 377 us.)
        int l1 = 0;
        uint32_t fw[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {                            // c0 + 4 c1
            const int b0 = k + 32 * side, b1 = b0 + 16;
            const int x0 = Hw[b0 * 32 + lane], y0 = Hw[b0 * 32 + (lane ^ 16)];
            const int x1 = Hw[b1 * 32 + lane], y1 = Hw[b1 * 32 + (lane ^ 16)];
            const int d0 = side ? y0 - x0 : x0 - y0, d1 = side ? y1 - x1 : x1 - y1;
            l1 += abs(d0) + abs(d1);
            fw[k] = pack_bf16((float)d0 * 0.125f, (float)d1 * 0.125f);
        }
        l1 += __shfl_xor_sync(FULL, l1, 16);
        const int lb = max(abs(m - nn), (l1 + 5) / 6);
        const int r0 = g, r1 = g + 8;
        const int m0 = __shfl_sync(FULL, m, r0), n0 = __shfl_sync(FULL, nn, r0);
        const int m1 = __shfl_sync(FULL, m, r1), n1 = __shfl_sync(FULL, nn, r1);
        float o[4];
        const int lb0 = __shfl_sync(FULL, lb, r0), lb1 = __shfl_sync(FULL, lb, r1);
        if constexpr (MODEL) {
            uint32_t* F = reinterpret_cast<uint32_t*>(hist_all + wib * 64 * 32);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 16; ++k) F[sl * RM_ROW + 8 * (k & 3) + 2 * (k >> 2) + side] = fw[k];
            F[sl * RM_ROW + 32 + 4 * side] = side ? 0u : pack_bf16(m * (1.0f / 256.0f), nn * (1.0f / 256.0f));
#pragma unroll
            for (int k = 1; k < 4; ++k) F[sl * RM_ROW + 32 + 4 * side + k] = 0u;
            __syncwarp();
            uint32_t a[TK1 / 16][4];
#pragma unroll
            for (int kt = 0; kt < TK1 / 16; ++kt) {
                a[kt][0] = F[r0 * RM_ROW + 8 * kt + tg];
                a[kt][1] = F[r1 * RM_ROW + 8 * kt + tg];
                a[kt][2] = F[r0 * RM_ROW + 8 * kt + tg + 4];
                a[kt][3] = F[r1 * RM_ROW + 8 * kt + tg + 4];
            }
            tc_tile_forward(S, a, o);
        } else {
            (void)fw;
            o[0] = o[1] = log2f((float)lb0 + 1.f);
            o[2] = o[3] = log2f((float)lb1 + 1.f);
        }
        if (tg == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = h ? r1 : r0;
                const int pr = tile * (16 >> lg) + (r >> lg);
                if (pr >= n || (r & ((1 << lg) - 1)) != 0) continue;
                const int mr = h ? m1 : m0, nr = h ? n1 : n0, lbr = h ? lb1 : lb0;
                const float y0 = h ? o[2] : o[0];
                const int it = route_item(mr, nr, D.pure[pr] != 0, D.pure[n + pr] != 0, lbr, y0, smax, lane_smax);
                item[pr] = it;
                if (lb_out) lb_out[pr] = lbr;
                if (y_out) { y_out[2 * (int64_t)pr] = y0; y_out[2 * (int64_t)pr + 1] = h ? o[3] : o[1]; }
                if (it < 0) {
                    out_score[pr] = -1;
                    if (out_len) out_len[pr] = 0;
                } else {
                    atomicAdd(&local[it & 0xff], 1);
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < 2 * ROUTE_BUCKETS && local[threadIdx.x]) atomicAdd(&counts[threadIdx.x], local[threadIdx.x]);
}

static size_t route_model_smem() { return sizeof(TcSmem) + (size_t)RM_WARPS * 64 * 32 * sizeof(int); }

// The fused routing pass over a WFA batch (D.packed and D.pure set): per pair
// the queue item, lower bound and prediction; bucket totals into counts.
// model = false: the queue items from the lower bound alone.
cudaError_t launch_route_model(const PairDesc& D, int smax, int lane_smax, bool model, int32_t* item, int32_t* lb,
                               float* y, int32_t* counts, int32_t* out_score, int32_t* out_len, cudaStream_t st)
{
    const __nv_bfloat16* w = cost_model_weights();
    if (model && !w) return cudaErrorNotReady;
    if (D.n <= 0) return cudaSuccess;
    if (const cudaError_t e = prepare_mlp()) return e;
    // Lanes to a side: as many as keep every tile a warp of its own.  One lane a side
    // leaves the 2,000 long pairs' counting to 125 warps (2,000 of 2-10 kb: pass 256 us,
    // with 16 lanes 47); the rows a tile then lacks cost nothing that waits.
    int lg = 0;
    while (lg < 4 && ((int64_t)D.n << (lg + 1)) <= (int64_t)16 * RM_WARPS * device_sms()) ++lg;
    int blocks = (int)((((int64_t)D.n << lg) + 16 * RM_WARPS - 1) / (16 * RM_WARPS));
    blocks = std::min(blocks, device_sms());
    launch_begin(K_MLP, st);
    auto kernel = model ? (lg ? route_model_kernel<true, true> : route_model_kernel<true, false>)
                        : (lg ? route_model_kernel<false, true> : route_model_kernel<false, false>);
    kernel<<<blocks, 32 * RM_WARPS, route_model_smem(), st>>>(w, D, smax, lane_smax, item, lb, y, counts, out_score,
                                                              out_len, lg);
    launch_end(K_MLP, st);
    return cudaGetLastError();
}

static cudaError_t run_forward_tc(const __nv_bfloat16* w, const float* feat, int n, float* y, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    if (const cudaError_t e = prepare_mlp()) return e;
    int blocks = (n + 127) / 128;
    blocks = std::min(blocks, device_sms() * 2);
    launch_begin(K_MLP, st);
    mlp_forward_tc_kernel<<<blocks, 256, sizeof(TcSmem), st>>>(w, feat, n, y);
    launch_end(K_MLP, st);
    return cudaGetLastError();
}

// --------------------------------------------------------- model state --
// One model per device: fp32 master, bf16 working copy, Adam moments, grads.
struct Model {
    float* master = nullptr;
    __nv_bfloat16* w = nullptr;
    float *m1 = nullptr, *m2 = nullptr, *grad = nullptr;   // grad: GRAD_COPIES copies; the loss behind the first
    int step = 0;
    bool ready = false;
};
// Two models per device, the same network: slot 0 the WFA cost model (edit
// distance and wavefront work), slot 1 the Smith-Waterman variant model (best
// score as a fraction of the all-match score).  The C API's set / get /
// forward / gradient / train calls act on the calling thread's selected slot
// (ga_model_select); each routing pass reads its own slot.
constexpr int N_MODEL_SLOTS = 2;
static std::mutex g_model_mu;
static Model g_models[16][N_MODEL_SLOTS];
static thread_local int t_model_slot = 0;

static Model* model_for(int slot, bool create)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) { cudaGetLastError(); return nullptr; }
    Model& M = g_models[dev][slot];
    if (!M.master && create) {
        if (cudaMalloc(&M.master, NPARAM * sizeof(float)) != cudaSuccess ||
            cudaMalloc(&M.w, NPARAM * sizeof(__nv_bfloat16)) != cudaSuccess ||
            cudaMalloc(&M.m1, NPARAM * sizeof(float)) != cudaSuccess ||
            cudaMalloc(&M.m2, NPARAM * sizeof(float)) != cudaSuccess ||
            cudaMalloc(&M.grad, GRAD_COPIES * GRAD_STRIDE * sizeof(float)) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
    }
    return M.master ? &M : nullptr;
}

// The shared-memory limits of this file's kernels, per device and outside any stream
// capture (prepare_mlp is called while planning a batch).
cudaError_t prepare_mlp()
{
    constexpr int MAX_DEV = 64;
    static std::mutex mu;
    static std::atomic<bool> ready[MAX_DEV];
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev >= 0 && dev < MAX_DEV;
    if (known && ready[dev].load(std::memory_order_acquire)) return cudaSuccess;
    std::lock_guard<std::mutex> lk(mu);
    auto limit = [](auto kernel, size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    cudaError_t r = limit(mlp_forward_kernel, sizeof(MlpSmem));
    if (r == cudaSuccess) r = limit(mlp_backward_kernel, sizeof(MlpSmem));
    if (r == cudaSuccess) r = limit(mlp_forward_tc_kernel, sizeof(TcSmem));
    for (auto kernel : {route_model_kernel<true, true>, route_model_kernel<true, false>,
                        route_model_kernel<false, true>, route_model_kernel<false, false>})
        if (r == cudaSuccess) r = limit(kernel, route_model_smem());
    if (known && r == cudaSuccess) ready[dev].store(true, std::memory_order_release);
    return r;
}

// A tile a block, no more blocks than multiprocessors (a block's shared memory fills one).
static int mlp_blocks(int n) { return std::min((int)(((int64_t)n + TILE - 1) / TILE), device_sms()); }

static cudaError_t run_forward(const __nv_bfloat16* w, const float* feat, int n, float* y, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    if (const cudaError_t e = prepare_mlp()) return e;
    launch_begin(K_MLP, st);
    mlp_forward_kernel<<<mlp_blocks(n), MLP_T, sizeof(MlpSmem), st>>>(w, feat, n, y);
    launch_end(K_MLP, st);
    return cudaGetLastError();
}

// grad: GRAD_COPIES copies of GRAD_STRIDE floats; the result is the first, the loss at NPARAM.
static cudaError_t run_backward(const __nv_bfloat16* w, const float* feat, const float* target, int n, float* grad,
                                cudaStream_t st)
{
    if (const cudaError_t e = prepare_mlp()) return e;
    cudaMemsetAsync(grad, 0, GRAD_COPIES * GRAD_STRIDE * sizeof(float), st);
    launch_begin(K_MLP, st);
    mlp_backward_kernel<<<mlp_blocks(n), MLP_T, sizeof(MlpSmem), st>>>(w, feat, target, n, 1.0f / (float)n, grad);
    launch_end(K_MLP, st);
    launch_begin(K_MLP, st);
    fold_grad_kernel<<<(NPARAM + 256) / 256, 256, 0, st>>>(grad);
    launch_end(K_MLP, st);
    return cudaGetLastError();
}

cudaError_t launch_sketch(const PairDesc& D, float* feat, int32_t* lb, cudaStream_t st, bool sw)
{
    if (D.n <= 0) return cudaSuccess;
    int blocks = (D.n + 7) / 8;
    blocks = std::min(blocks, device_sms() * 16);
    // WFA pairs (150-10,000 bases): differences / 8, lengths / 256; SW pairs
    // (text with flanks, up to tens of kb): differences / 64, lengths / 8192
    const float s_diff = sw ? 1.0f / 64.0f : 0.125f, s_len = sw ? 1.0f / 8192.0f : 1.0f / 256.0f;
    launch_begin(K_SKETCH, st);
    if (D.packed) sketch_packed_kernel<<<blocks, 256, 0, st>>>(D, feat, lb, s_diff, s_len);
    else sketch_kernel<<<blocks, 256, 0, st>>>(D, feat, lb, s_diff, s_len);
    launch_end(K_SKETCH, st);
    return cudaGetLastError();
}

static Model* model_for_current(bool create) { return model_for(t_model_slot, create); }

// A slot's weights on the current device for inference, or null when none is loaded.
static const __nv_bfloat16* model_weights(int slot)
{
    std::lock_guard<std::mutex> lk(g_model_mu);
    Model* M = model_for(slot, false);
    return (M && M->ready) ? M->w : nullptr;
}
const __nv_bfloat16* cost_model_weights() { return model_weights(0); }

bool cost_model_loaded() { return cost_model_weights() != nullptr; }
bool sw_model_loaded() { return model_weights(1) != nullptr; }

// Inference of the selected slot's model: the tensor-core forward pass.
cudaError_t launch_mlp_forward(const float* feat, int n, float* y, cudaStream_t st)
{
    const __nv_bfloat16* w = model_weights(t_model_slot);
    if (!w) return cudaErrorNotReady;
    return run_forward_tc(w, feat, n, y, st);
}

// SW variant routing: features of every pair (a = text, b = pattern), the
// SW model's prediction of the best score as a fraction of the all-match
// score match * min(m, n), and try16[p] = 1 for a pair the 16-bit kernel
// should try: its predicted score with a margin (x 1.15 + 8 matches) fits 16
// bits (sw16_eligible_opt's test).  Purity and the exact hand-over at the
// 16-bit limit are the planner's and the kernel's, so a wrong prediction only
// costs time.
__global__ void sw_route_kernel(PairDesc D, const float* __restrict__ y, int match, int go, uint8_t* __restrict__ try16)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.n; p += gridDim.x * blockDim.x) {
        const int m = D.a_len[p], n = D.b_len[p];
        const float frac = fminf(fmaxf(y[2 * (int64_t)p], 0.f), 1.f);
        const float all = (float)match * (float)min(max(m, 0), max(n, 0));
        const float pred = frac * all * 1.15f + 8.f * (float)match;
        try16[p] = (m > 0 && n > 0 && pred + (float)(BIAS16 + go) < 32000.f) ? 1 : 0;
    }
}

cudaError_t launch_sw_route(const PairDesc& D, int match, int go, float* feat, float* y, uint8_t* try16, cudaStream_t st)
{
    const __nv_bfloat16* w = model_weights(1);
    if (!w) return cudaErrorNotReady;
    if (D.n <= 0) return cudaSuccess;
    cudaError_t e = launch_sketch(D, feat, nullptr, st, true);
    if (e == cudaSuccess) e = run_forward_tc(w, feat, D.n, y, st);
    if (e != cudaSuccess) return e;
    int blocks = std::min((D.n + 255) / 256, device_sms() * 8);
    launch_begin(K_ROUTE, st);
    sw_route_kernel<<<blocks, 256, 0, st>>>(D, y, match, go, try16);
    launch_end(K_ROUTE, st);
    return cudaGetLastError();
}

}  // namespace ga

using namespace ga;

extern "C" {

int32_t ga_cost_model_nparams(void) { return NPARAM; }

int32_t ga_model_select(int32_t which)
{
    if (which < 0 || which >= N_MODEL_SLOTS) return GA_INVALID_ARGUMENT;
    t_model_slot = which;
    return GA_OK;
}

int32_t ga_cost_model_set(const float* params, int32_t n)
{
    if (!params || n != NPARAM) return GA_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(g_model_mu);
    Model* M = model_for_current(true);
    if (!M) return GA_DEVICE_ERROR;
    if (cudaMemcpy(M->master, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(M->m1, 0, NPARAM * sizeof(float)) != cudaSuccess ||
        cudaMemset(M->m2, 0, NPARAM * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        return GA_DEVICE_ERROR;
    }
    launch_begin(K_MLP, nullptr);
    to_bf16_kernel<<<64, 256>>>(M->master, M->w, NPARAM);
    launch_end(K_MLP, nullptr);
    if (cudaDeviceSynchronize() != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    M->step = 0;
    M->ready = true;
    return GA_OK;
}

int32_t ga_cost_model_get(float* params, int32_t n)
{
    if (!params || n != NPARAM) return GA_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(g_model_mu);
    Model* M = model_for_current(false);
    if (!M || !M->ready) return GA_INVALID_ARGUMENT;
    if (cudaMemcpy(params, M->master, NPARAM * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess) {
        cudaGetLastError();
        return GA_DEVICE_ERROR;
    }
    return GA_OK;
}

int32_t ga_wfa_features(const ga_device_batch* b, float* feat, int32_t* lower_bound, void* stream)
{
    if (!b || b->n < 0 || !feat) return GA_INVALID_ARGUMENT;
    PairDesc D;
    D.seq = b->seq; D.packed = nullptr; D.pure = nullptr;
    D.a_off = b->a_off; D.a_len = b->a_len; D.b_off = b->b_off; D.b_len = b->b_len; D.out_off = b->out_off; D.n = b->n;
    cudaStream_t st = (cudaStream_t)stream;
    if (launch_sketch(D, feat, lower_bound, st, false) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    if (!stream && cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    return GA_OK;
}

int32_t ga_sw_features(const ga_device_batch* b, float* feat, void* stream)
{
    if (!b || b->n < 0 || !feat) return GA_INVALID_ARGUMENT;
    PairDesc D;
    D.seq = b->seq; D.packed = nullptr; D.pure = nullptr;
    D.a_off = b->a_off; D.a_len = b->a_len; D.b_off = b->b_off; D.b_len = b->b_len; D.out_off = b->out_off; D.n = b->n;
    cudaStream_t st = (cudaStream_t)stream;
    if (launch_sketch(D, feat, nullptr, st, true) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    if (!stream && cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    return GA_OK;
}

int32_t ga_mlp_forward(const float* feat, int32_t n, float* y, void* stream)
{
    if (!feat || !y || n < 0) return GA_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* w = model_weights(t_model_slot);
    if (!w) return GA_INVALID_ARGUMENT;
    const cudaError_t e = run_forward(w, feat, n, y, st);
    if (e == cudaErrorNotReady) return GA_INVALID_ARGUMENT;
    if (e != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    if (!stream && cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    return GA_OK;
}

int32_t ga_mlp_forward_fast(const float* feat, int32_t n, float* y, void* stream)
{
    if (!feat || !y || n < 0) return GA_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const cudaError_t e = launch_mlp_forward(feat, n, y, st);
    if (e == cudaErrorNotReady) return GA_INVALID_ARGUMENT;
    if (e != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    if (!stream && cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    return GA_OK;
}

int32_t ga_mlp_gradient(const float* feat, const float* target, int32_t n, float* grad_host, float* loss_host)
{
    if (!feat || !target || n <= 0 || !grad_host) return GA_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(g_model_mu);
    Model* M = model_for_current(false);
    if (!M || !M->ready) return GA_INVALID_ARGUMENT;
    if (run_backward(M->w, feat, target, n, M->grad, 0) != cudaSuccess ||
        cudaMemcpy(grad_host, M->grad, NPARAM * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess ||
        (loss_host && cudaMemcpy(loss_host, M->grad + NPARAM, sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)) {
        cudaGetLastError();
        return GA_DEVICE_ERROR;
    }
    return GA_OK;
}

int32_t ga_mlp_train_step(const float* feat, const float* target, int32_t n, float lr, float* loss_host, void* stream)
{
    if (!feat || !target || n <= 0) return GA_INVALID_ARGUMENT;
    std::lock_guard<std::mutex> lk(g_model_mu);
    Model* M = model_for_current(false);
    if (!M || !M->ready) return GA_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (run_backward(M->w, feat, target, n, M->grad, st) != cudaSuccess) { cudaGetLastError(); return GA_DEVICE_ERROR; }
    M->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f / (1.f - powf(b1, (float)M->step)), c2 = 1.f / (1.f - powf(b2, (float)M->step));
    launch_begin(K_MLP, st);
    adam_kernel<<<64, 256, 0, st>>>(M->master, M->w, M->grad, M->m1, M->m2, NPARAM, lr, b1, b2, 1e-8f, c1, c2);
    launch_end(K_MLP, st);
    if (cudaGetLastError() != cudaSuccess) return GA_DEVICE_ERROR;
    if (loss_host) {
        if (cudaMemcpyAsync(loss_host, M->grad + NPARAM, sizeof(float), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            cudaGetLastError();
            return GA_DEVICE_ERROR;
        }
        *loss_host /= (float)n;
    }
    return GA_OK;
}

}  // extern "C"
