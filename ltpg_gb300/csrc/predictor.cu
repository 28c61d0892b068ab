// predictor.cu — contention predictor: which key-hash buckets to stage.
//
// Input per bucket: log1p of its registration counts in the last 4 batches
// (counted by the tuned execute kernels).  Model: MLP 4 -> 64 -> 64 -> 1 with
// ReLU, BF16 weights and activations, FP32 accumulation; the output predicts
// log1p of the bucket's count in the next batch.  After every batch:
//   roll      the batch's counts enter a 5-batch ring and the counters reset;
//   train     one Adam step on 4,096 buckets (a rotating 1/16 of them): the
//             features are batches t-5..t-2, the label batch t-1 (the "previous
//             batch's registration contention");
//   infer     all 65,536 buckets from batches t-4..t-1;
//   select    the top-k scores become the staged set (k = staging groups).
// Six kernels per batch: roll (+ ring advance), training forward, fused
// backward (+ loss), Adam (+ BF16 copies), inference forward, select (+ step
// counters).
// The forward pass runs on the tensor cores (mma.sync m16n8k16, BF16 inputs,
// FP32 accumulators); backward and Adam are FP32.  The predictor only picks
// the staged set, which changes speed, never a commit decision.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <cstring>
#include <vector>

#include "stage.cuh"

namespace ltpg {

namespace cg = cooperative_groups;

constexpr int PH = 64;            // hidden width
constexpr int PF = 4;             // features (batches of history)
constexpr int P_RING = 5;         // count ring: 4 feature batches + 1 label batch
constexpr int P_TRAIN = 4096;     // samples per training step
constexpr int P_W1 = 0, P_B1 = P_W1 + PH * PF, P_W2 = P_B1 + PH, P_B2 = P_W2 + PH * PH, P_W3 = P_B2 + PH,
              P_B3 = P_W3 + PH, P_NPARAM = P_B3 + 1;  // packed FP32 parameter layout

struct PredDev {
    float *param, *m, *v, *grad;          // P_NPARAM each
    __nv_bfloat16 *w1b, *w2b;             // BF16 copies: w1b [64][16] (K padded), w2b [64][64]
    uint32_t *ring;                       // P_RING x buckets
    float *scores;                        // buckets
    float *act;                           // training activations: X [S][4], H1 [S][64], H2 [S][64], Y [S], T [S]
    uint32_t *state;                      // [0] ring position, [1] step, [2] batches seen, [3] blocks done
    float *loss;                          // [0] last training loss, [1] its running sum over sample tiles
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ void mma_bf16(float *d, const uint32_t *a, const uint32_t *b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Feature f of bucket b: log1p of its count in the f-th of the 4 ring slots
// ending at `newest` (oldest first).
__device__ __forceinline__ float feature(const uint32_t *ring, uint32_t newest, uint32_t b, uint32_t f) {
    const uint32_t slot = (newest + P_RING - (PF - 1 - f)) % P_RING;
    return log1pf((float)ring[slot * STAGE_BUCKETS + b]);
}

// ---- forward on tensor cores ----------------------------------------------------
// A warp runs 16 samples at a time.  Layer 1: [16 x 16] (4 features, zero
// padded) x W1^T -> 8 n-tiles of 8; the FP32 accumulators of tiles 2kb and
// 2kb+1, after bias + ReLU + BF16 rounding, are exactly the A fragment of
// k-block kb of layer 2 (16 x 64 x 64, 32 mma).  Layer 3 is a dot product
// reduced over the 4 lanes that share a row.
// mode 0: inference over `n` buckets (x from the ring, newest = slot t-1),
//         writes scores.  mode 1: training samples (x from slots t-5..t-2),
//         also stores X, H1, H2, Y, T for the backward pass.
// mode 2: x given in `xin` [n][4] (tests), writes y.  mode 3: x given in `xin`,
//         stores X, H1, H2, Y like mode 1 (the gradient test sets T).
// A warp has little to do, so what surrounds it bounds it: the weights come in
// 16-byte loads, their rows are padded so that the eight rows of a fragment lie
// in different banks (unpadded they met in one), and the four lanes of a row
// take one feature each (each took all four).  One tile a warp.  65,536 buckets
// 20 -> 11 us, 4,096 samples 14 -> 9.4 us (cold).
constexpr int W1_ROW = 24, W2_ROW = 72;  // padded rows in shared memory, BF16
__global__ void __launch_bounds__(256) pred_forward(PredDev p, uint32_t n, int mode, const float *__restrict__ xin,
                                                    float *__restrict__ yout) {
    __shared__ __align__(16) __nv_bfloat16 w1s[PH * W1_ROW];
    __shared__ __align__(16) __nv_bfloat16 w2s[PH * W2_ROW];
    __shared__ float b1s[PH], b2s[PH], w3s[PH];
    __shared__ float b3s;
    for (int i = threadIdx.x; i < PH * 2; i += blockDim.x)
        *reinterpret_cast<uint4 *>(w1s + i / 2 * W1_ROW + i % 2 * 8) = reinterpret_cast<const uint4 *>(p.w1b)[i];
    for (int i = threadIdx.x; i < PH * PH / 8; i += blockDim.x)
        *reinterpret_cast<uint4 *>(w2s + i / 8 * W2_ROW + i % 8 * 8) = reinterpret_cast<const uint4 *>(p.w2b)[i];
    for (int i = threadIdx.x; i < PH; i += blockDim.x) {
        b1s[i] = p.param[P_B1 + i];
        b2s[i] = p.param[P_B2 + i];
        w3s[i] = p.param[P_W3 + i];
    }
    if (threadIdx.x == 0) b3s = p.param[P_B3];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const uint32_t pos = p.state[0], step = p.state[1];
    const uint32_t newest = (pos + P_RING - 1) % P_RING;  // slot of batch t-1
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t s0 = warp * 16; s0 < n; s0 += n_warps * 16) {
        // sample ids of rows g and g + 8
        uint32_t sid[2] = {s0 + g, s0 + g + 8};
        float xq[2], tr[2] = {0.f, 0.f};  // this lane's feature (q) of both rows
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t s = sid[h];
            xq[h] = 0.f;
            if (s >= n) continue;
            if (mode == 2 || mode == 3) {
                xq[h] = xin[s * PF + q];
            } else if (mode == 1) {
                const uint32_t b = (s * 16u + (step & 15u)) & (STAGE_BUCKETS - 1u);  // rotating 1/16 of buckets
                xq[h] = feature(p.ring, (newest + P_RING - 1) % P_RING, b, q);
                if (q == 0) tr[h] = log1pf((float)p.ring[newest * STAGE_BUCKETS + b]);
            } else {
                xq[h] = feature(p.ring, newest, s, q);
            }
        }
        // A fragment of layer 1: features are k = 0..3 (lanes q = 0, 1)
        uint32_t a1[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float lo = __shfl_sync(FULL, xq[h], (lane & 28u) | ((2u * q) & 3u));
            const float hi = __shfl_sync(FULL, xq[h], (lane & 28u) | ((2u * q + 1u) & 3u));
            a1[h] = q < 2u ? pack_bf16(lo, hi) : 0u;
        }
        a1[2] = 0u;
        a1[3] = 0u;
        float h1[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            h1[nt][0] = h1[nt][1] = h1[nt][2] = h1[nt][3] = 0.f;
            const __nv_bfloat16 *wr = w1s + (nt * 8 + g) * W1_ROW;
            uint32_t b[2] = {*reinterpret_cast<const uint32_t *>(wr + q * 2),
                             *reinterpret_cast<const uint32_t *>(wr + 8 + q * 2)};
            mma_bf16(h1[nt], a1, b);
            const int c = nt * 8 + q * 2;
            h1[nt][0] = fmaxf(h1[nt][0] + b1s[c], 0.f);
            h1[nt][1] = fmaxf(h1[nt][1] + b1s[c + 1], 0.f);
            h1[nt][2] = fmaxf(h1[nt][2] + b1s[c], 0.f);
            h1[nt][3] = fmaxf(h1[nt][3] + b1s[c + 1], 0.f);
        }
        float h2[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) h2[nt][0] = h2[nt][1] = h2[nt][2] = h2[nt][3] = 0.f;
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
            uint32_t a[4] = {pack_bf16(h1[2 * kb][0], h1[2 * kb][1]), pack_bf16(h1[2 * kb][2], h1[2 * kb][3]),
                             pack_bf16(h1[2 * kb + 1][0], h1[2 * kb + 1][1]),
                             pack_bf16(h1[2 * kb + 1][2], h1[2 * kb + 1][3])};
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const __nv_bfloat16 *wr = w2s + (nt * 8 + g) * W2_ROW + kb * 16;
                uint32_t b[2] = {*reinterpret_cast<const uint32_t *>(wr + q * 2),
                                 *reinterpret_cast<const uint32_t *>(wr + 8 + q * 2)};
                mma_bf16(h2[nt], a, b);
            }
        }
        float y0 = 0.f, y1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int c = nt * 8 + q * 2;
            h2[nt][0] = fmaxf(h2[nt][0] + b2s[c], 0.f);
            h2[nt][1] = fmaxf(h2[nt][1] + b2s[c + 1], 0.f);
            h2[nt][2] = fmaxf(h2[nt][2] + b2s[c], 0.f);
            h2[nt][3] = fmaxf(h2[nt][3] + b2s[c + 1], 0.f);
            y0 += h2[nt][0] * w3s[c] + h2[nt][1] * w3s[c + 1];
            y1 += h2[nt][2] * w3s[c] + h2[nt][3] * w3s[c + 1];
        }
        y0 += __shfl_xor_sync(FULL, y0, 1);
        y0 += __shfl_xor_sync(FULL, y0, 2);
        y1 += __shfl_xor_sync(FULL, y1, 1);
        y1 += __shfl_xor_sync(FULL, y1, 2);
        y0 += b3s;
        y1 += b3s;
        if (mode == 1 || mode == 3) {
            float *X = p.act, *H1 = X + P_TRAIN * PF, *H2 = H1 + P_TRAIN * PH, *Y = H2 + P_TRAIN * PH,
                  *T = Y + P_TRAIN;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t s = sid[h];
                if (s >= n) continue;
                X[s * PF + q] = xq[h];
                if (q == 0) {
                    Y[s] = h ? y1 : y0;
                    if (mode == 1) T[s] = tr[h];
                }
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    const int c = nt * 8 + q * 2;
                    // layer 2 consumed BF16(h1): keep that value for the gradient
                    *reinterpret_cast<float2 *>(H1 + s * PH + c) =
                        make_float2(__bfloat162float(__float2bfloat16_rn(h1[nt][2 * h])),
                                    __bfloat162float(__float2bfloat16_rn(h1[nt][2 * h + 1])));
                    *reinterpret_cast<float2 *>(H2 + s * PH + c) = make_float2(h2[nt][2 * h], h2[nt][2 * h + 1]);
                }
            }
        } else if (q == 0) {
            float *out = mode == 2 ? yout : p.scores;
            if (sid[0] < n) out[sid[0]] = y0;
            if (sid[1] < n) out[sid[1]] = y1;
        }
    }
}

// ---- backward (FP32) ----------------------------------------------------------------
// grad layout = packed params.  Loss = mean over samples of (y - t)^2.
// dz2[s][j] = 2 (y - t) / S * w3[j] * [h2 > 0];  dh1[s][k] = sum_j dz2[s][j] W2[j][k];
// dz1 = dh1 * [h1 > 0].  The weights used are the BF16 copies the forward used.
// One kernel: a block walks tiles of PB samples; per tile dz2 and dz1 are made
// in shared memory, and each thread adds the tile's terms of its parameters to
// registers: a 4 x 4 block of W2, one of W1 and at most one of the others.  The
// block adds its sums to the global gradient once at the end, and its share of
// the squared error to loss[1].  Shared-memory reads bound it: the 4 x 4 block
// reads two 16-byte vectors for 16 products, where one parameter at a time read
// two words for each (4,096 samples 36 -> 11 us).
constexpr int PB = 16;       // samples per tile
constexpr int PR = PH + 4;   // padded row of a tile

__global__ void __launch_bounds__(256) pred_backward(PredDev p, uint32_t S) {
    const float *X = p.act, *H1 = X + P_TRAIN * PF, *H2 = H1 + P_TRAIN * PH, *Y = H2 + P_TRAIN * PH, *T = Y + P_TRAIN;
    __shared__ __align__(16) float w2[PH * PH];
    __shared__ __align__(16) float d2[PB * PR], d1[PB * PR], h1[PB * PR], h2[PB * PR];
    __shared__ float xs[PB][PF], dys[PB];
    const uint32_t tid = threadIdx.x;
    auto at = [](float *row, uint32_t c) { return reinterpret_cast<float4 *>(row + c); };
    for (uint32_t i = tid; i < PH * PH / 2; i += blockDim.x) {
        const float2 w = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162 *>(p.w2b)[i]);
        w2[2 * i] = w.x;
        w2[2 * i + 1] = w.y;
    }
    // this thread's element of a tile, its 4 x 4 block of W2, its W1 parameter
    const uint32_t r0 = tid / 16u, c0 = tid % 16u * 4u;
    const float4 w3 = make_float4(p.param[P_W3 + c0], p.param[P_W3 + c0 + 1], p.param[P_W3 + c0 + 2], p.param[P_W3 + c0 + 3]);
    float acc2[4][4] = {}, acc1 = 0.f, acco = 0.f, lacc = 0.f;
    const uint32_t n_tiles = (S + PB - 1) / PB;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t s0 = tile * PB, s = s0 + r0;
        float4 v1 = make_float4(0.f, 0.f, 0.f, 0.f), v2 = v1;
        float e = 0.f;
        if (s < S) {
            v1 = *reinterpret_cast<const float4 *>(H1 + s * PH + c0);
            v2 = *reinterpret_cast<const float4 *>(H2 + s * PH + c0);
            e = Y[s] - T[s];
        }
        const float dy = 2.f * e / (float)S;
        __syncthreads();  // w2 loaded, or the previous tile consumed
        *at(h1 + r0 * PR, c0) = v1;
        *at(h2 + r0 * PR, c0) = v2;
        *at(d2 + r0 * PR, c0) = make_float4(v2.x > 0.f ? dy * w3.x : 0.f, v2.y > 0.f ? dy * w3.y : 0.f,
                                            v2.z > 0.f ? dy * w3.z : 0.f, v2.w > 0.f ? dy * w3.w : 0.f);
        if (c0 == 0u) {
            dys[r0] = dy;
            lacc += e * e;
        }
        if (tid < PB * PF) {  // layer 1 consumed BF16(x)
            const uint32_t sx = s0 + tid / PF;
            xs[tid / PF][tid % PF] = sx < S ? __bfloat162float(__float2bfloat16_rn(X[sx * PF + tid % PF])) : 0.f;
        }
        __syncthreads();
        {  // dz1 of sample r0, units c0 .. c0 + 3
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (uint32_t j4 = 0; j4 < PH; j4 += 4) {
                const float4 d = *at(d2 + r0 * PR, j4);
                const float dj[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const float4 w = *at(w2 + (j4 + i) * PH, c0);
                    a.x += dj[i] * w.x;
                    a.y += dj[i] * w.y;
                    a.z += dj[i] * w.z;
                    a.w += dj[i] * w.w;
                }
            }
            *at(d1 + r0 * PR, c0) = make_float4(v1.x > 0.f ? a.x : 0.f, v1.y > 0.f ? a.y : 0.f, v1.z > 0.f ? a.z : 0.f,
                                                v1.w > 0.f ? a.w : 0.f);
        }
        float a2[4][4] = {};
#pragma unroll 4
        for (int r = 0; r < PB; ++r) {
            const float4 d = *at(d2 + r * PR, r0 * 4u), h = *at(h1 + r * PR, c0);
            const float dj[4] = {d.x, d.y, d.z, d.w}, hk[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) a2[j][k] += dj[j] * hk[k];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc2[j][k] += a2[j][k];
        float ao = 0.f;  // b2, w3, b3
        if (tid < PH)
            for (int r = 0; r < PB; ++r) ao += d2[r * PR + tid];
        else if (tid < 2 * PH)
            for (int r = 0; r < PB; ++r) ao += dys[r] * h2[r * PR + tid - PH];
        else if (tid == 2 * PH)
            for (int r = 0; r < PB; ++r) ao += dys[r];
        __syncthreads();
        float a1 = 0.f;
        for (int r = 0; r < PB; ++r) a1 += d1[r * PR + tid / PF] * xs[r][tid % PF];
        acc1 += a1;
        if (tid >= 192u)  // b1
            for (int r = 0; r < PB; ++r) ao += d1[r * PR + tid - 192u];
        acco += ao;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
        atomicAdd(reinterpret_cast<float4 *>(p.grad + P_W2 + (r0 * 4u + j) * PH + c0),
                  make_float4(acc2[j][0], acc2[j][1], acc2[j][2], acc2[j][3]));
    atomicAdd(&p.grad[P_W1 + tid], acc1);
    const int other = tid < PH ? P_B2 + (int)tid : tid < 2 * PH ? P_W3 + (int)tid - PH
                      : tid == 2 * PH ? P_B3 : tid >= 192u ? P_B1 + (int)tid - 192 : -1;
    if (other >= 0) atomicAdd(&p.grad[other], acco);
    // the squared errors of the tiles' rows, one per 16 threads
    lacc += __shfl_xor_sync(FULL, lacc, 16);
    __syncthreads();  // dys is read to the end of the last tile
    if ((tid & 31u) == 0u) dys[tid >> 5] = lacc;
    __syncthreads();
    if (tid == 0) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += dys[w];
        atomicAdd(&p.loss[1], t);
    }
}
static_assert(P_W2 % 4 == 0 && PH == 64 && PF == 4, "the layout of a thread's parameters");

// Adam (Kingma & Ba, 2015) on the FP32 master parameters; each updated weight
// of W1 / W2 is also written to its BF16 copy (the zero padding of W1's K
// dimension is written once, by pred_cast).  The first thread turns the
// summed squared error into the step's loss.
__global__ void pred_adam(PredDev p, float lr, uint32_t S) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const uint32_t t = p.state[1] + 1;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P_NPARAM; i += gridDim.x * blockDim.x) {
        const float g = p.grad[i];
        const float m = b1 * p.m[i] + (1.f - b1) * g;
        const float v = b2 * p.v[i] + (1.f - b2) * g * g;
        p.m[i] = m;
        p.v[i] = v;
        const float w = p.param[i] - lr * (m / c1) / (sqrtf(v / c2) + eps);
        p.param[i] = w;
        p.grad[i] = 0.f;
        if (i < (uint32_t)P_B1) p.w1b[(i / PF) * 16 + i % PF] = __float2bfloat16_rn(w);
        else if (i >= (uint32_t)P_W2 && i < (uint32_t)P_B2) p.w2b[i - P_W2] = __float2bfloat16_rn(w);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.loss[0] = p.loss[1] / (float)S;
        p.loss[1] = 0.f;
    }
}

// BF16 copies of W1 (K padded to 16) and W2 for the forward pass.
__global__ void pred_cast(PredDev p) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < PH * 16 + PH * PH; i += gridDim.x * blockDim.x) {
        if (i < PH * 16) {
            const uint32_t j = i / 16, k = i % 16;
            p.w1b[i] = __float2bfloat16_rn(k < PF ? p.param[P_W1 + j * PF + k] : 0.f);
        } else {
            p.w2b[i - PH * 16] = __float2bfloat16_rn(p.param[P_W2 + (i - PH * 16)]);
        }
    }
}

__global__ void pred_step_done(PredDev p, int trained) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        if (trained) p.state[1] += 1;
        p.state[2] += 1;
    }
}

// The batch's counts enter the ring and the counters restart for the next
// batch; the last block to finish advances the ring position.
__global__ void pred_roll(PredDev p, uint32_t *__restrict__ counts) {
    const uint32_t pos = p.state[0];
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < STAGE_BUCKETS; b += gridDim.x * blockDim.x) {
        p.ring[pos * STAGE_BUCKETS + b] = counts[b];
        counts[b] = 0u;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&p.state[3], 1u) == gridDim.x - 1u) {
            p.state[3] = 0u;
            p.state[0] = (pos + 1) % P_RING;
        }
    }
}

// Top-k scores -> staged set, in one cluster of eight blocks of 1024 threads,
// eight buckets to a thread.  Each score becomes a 16-bit order-preserving key
// (sign, exponent and 7 mantissa bits) in a register: two 256-bin histogram
// passes find the k-th largest key (one shared atomic per distinct bin of a
// warp; the blocks read one another's histograms); buckets above it are taken,
// then ties in bucket order until k.  Outputs: the bitmap and per-word ranks
// and the bucket -> group map.  The first thread also ends the predictor step
// (training step count when `trained`, batches seen).  (One block of 64 buckets
// to a thread, its keys in shared memory: 45 to 72 us; the cluster: 10 to 15.)
constexpr uint32_t SEL_BLOCKS = 8u;
static_assert(SEL_BLOCKS * 1024u * 8u == STAGE_BUCKETS, "eight buckets to a thread");

__global__ void __cluster_dims__(SEL_BLOCKS, 1, 1) __launch_bounds__(1024)
    pred_select(PredDev p, uint32_t k, uint32_t *__restrict__ bits, uint32_t *__restrict__ rank,
                uint16_t *__restrict__ map, int trained) {
    __shared__ uint32_t hist[2][256], all[256];
    __shared__ uint32_t sel_bin, sel_rem, total;
    __shared__ uint32_t wsum[32];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, me = cluster.block_rank();
    const uint32_t b0 = (me * 1024u + tid) * 8u;
    auto okey16 = [](float f) {
        const uint32_t u = __float_as_uint(f);
        return ((u & 0x80000000u) ? ~u : (u | 0x80000000u)) >> 16;
    };
    const float4 f0 = reinterpret_cast<const float4 *>(p.scores + b0)[0],
                 f1 = reinterpret_cast<const float4 *>(p.scores + b0)[1];
    const uint32_t key[8] = {okey16(f0.x), okey16(f0.y), okey16(f0.z), okey16(f0.w),
                             okey16(f1.x), okey16(f1.y), okey16(f1.z), okey16(f1.w)};
    if (tid < 256u) hist[0][tid] = hist[1][tid] = 0u;
    __syncthreads();
    // two passes: the high byte of the k-th largest key, then its low byte
    uint32_t hi = 0, remaining = k;
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool in = pass == 0 || (key[i] >> 8) == hi;
            const uint32_t bin = !in ? 256u : pass == 0 ? key[i] >> 8 : key[i] & 255u;
            const unsigned peers = __match_any_sync(FULL, bin);
            if (in && lane == (uint32_t)__ffs(peers) - 1u) atomicAdd(&hist[pass][bin], (uint32_t)__popc(peers));
        }
        cluster.sync();
        if (tid < 256u) {
            uint32_t sum = 0;
#pragma unroll
            for (uint32_t r = 0; r < SEL_BLOCKS; ++r) sum += *cluster.map_shared_rank(&hist[pass][tid], r);
            all[tid] = sum;
        }
        __syncthreads();
        if (tid < 32) {  // the bin holding the remaining-th largest key: warp-wide suffix sums
            const uint32_t lo = (31u - tid) * 8u;  // lane 0 holds the highest bins
            uint32_t c[8], tot = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) tot += (c[i] = all[lo + i]);
            const uint32_t incl = (uint32_t)warp_incl_scan((int)tot);  // keys in this lane's bins and all higher ones
            const uint32_t above = incl - tot;                        // keys in higher lanes' bins
            if (above < remaining && incl >= remaining) {
                uint32_t acc = above, bin = lo;
                for (int i = 7; i >= 0; --i) {
                    if (acc + c[i] >= remaining) {
                        bin = lo + (uint32_t)i;
                        break;
                    }
                    acc += c[i];
                }
                sel_bin = bin;
                sel_rem = remaining - acc;
            }
        }
        __syncthreads();
        hi = pass == 0 ? sel_bin : (hi << 8) | sel_bin;
        remaining = sel_rem;
    }
    // hi: the k-th largest key; `remaining` of the buckets with that key are
    // still needed, taken in bucket order.  Scan of (taken outright << 16 | ties)
    // over the block's threads, then the blocks before.
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) mine += key[i] > hi ? 0x10000u : key[i] == hi ? 1u : 0u;
    const uint32_t incl = (uint32_t)warp_incl_scan((int)mine);
    if (lane == 31u) wsum[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32) {
        const uint32_t w = wsum[tid], wi = (uint32_t)warp_incl_scan((int)w);
        wsum[tid] = wi - w;
        if (tid == 31) total = wi;
    }
    cluster.sync();
    uint32_t gt = 0, ties = 0;  // of the buckets before this thread's
#pragma unroll
    for (uint32_t r = 0; r < SEL_BLOCKS; ++r) {
        const uint32_t t = r < me ? *cluster.map_shared_rank(&total, r) : 0u;
        gt += t >> 16;
        ties += t & 0xFFFFu;
    }
    const uint32_t before = wsum[tid >> 5] + incl - mine;
    gt += before >> 16;
    ties += before & 0xFFFFu;
    const uint32_t r0 = gt + min(ties, remaining);
    uint32_t group = r0, mask = 0, m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool take = key[i] > hi || (key[i] == hi && ties++ < remaining);
        mask |= take ? 1u << i : 0u;
        m[i] = take ? group++ : STAGE_NONE;
    }
    reinterpret_cast<uint4 *>(map + b0)[0] =
        make_uint4(m[0] | m[1] << 16, m[2] | m[3] << 16, m[4] | m[5] << 16, m[6] | m[7] << 16);
    // a bitmap word is four threads'
    uint32_t word = mask << (8u * (tid & 3u));
    word |= __shfl_xor_sync(FULL, word, 1);
    word |= __shfl_xor_sync(FULL, word, 2);
    if ((tid & 3u) == 0u) {
        bits[b0 >> 5] = word;
        rank[b0 >> 5] = r0;
    }
    if (b0 == 0u) {
        if (trained) p.state[1] += 1;
        p.state[2] += 1;
    }
    cluster.sync();  // no block leaves while another reads its shared memory
}

}  // namespace ltpg

using namespace ltpg;

struct ltpg_predictor_state {
    PredDev d{};
    float *io = nullptr;  // test io buffer
    float lr = 3e-3f;
    uint32_t train_every = 1;
    uint64_t steps_host = 0;
};

namespace {
int pfail(ltpg_ctx *c, const char *msg) {
    c->err = msg;
    return LTPG_ERR_CUDA;
}
#define PCK(call)                                                 \
    do {                                                          \
        if ((call) != cudaSuccess) return pfail(c, #call " failed"); \
    } while (0)

// Xavier-uniform initial weights from a splitmix64 stream, biases 0.
void init_params(std::vector<float> &w, uint64_t seed) {
    w.assign(P_NPARAM, 0.f);
    uint64_t s = seed;
    auto uni = [&]() {
        s += 0x9E3779B97F4A7C15ull;
        uint64_t z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (float)((double)(z >> 11) * 0x1.0p-53 * 2.0 - 1.0);
    };
    const float a1 = sqrtf(6.f / (PF + PH)), a2 = sqrtf(6.f / (PH + PH)), a3 = sqrtf(6.f / (PH + 1));
    for (int i = 0; i < PH * PF; ++i) w[P_W1 + i] = a1 * uni();
    for (int i = 0; i < PH * PH; ++i) w[P_W2 + i] = a2 * uni();
    for (int i = 0; i < PH; ++i) w[P_W3 + i] = a3 * uni();
    for (int i = 0; i < PH; ++i) w[P_B1 + i] = 0.01f;
    for (int i = 0; i < PH; ++i) w[P_B2 + i] = 0.01f;
}
}  // namespace

extern "C" {

int ltpg_predictor_enable(ltpg_ctx *c, const ltpg_predictor_cfg *cfg) {
    if (!c || !cfg) return LTPG_ERR_INVALID;
    if (!cfg->enable) {
        c->pred_on = 0;
        c->stage_on = 0;
        drop_graphs_ctx(c);
        return LTPG_OK;
    }
    if (!c->stage_map) {
        const uint32_t none = 0;
        int r = ltpg_stage_set(c, &none, 1);  // allocates the stage arrays
        if (r) return r;
    }
    if (!c->pred) {
        ltpg_predictor_state *P = new ltpg_predictor_state();
        c->pred = P;
        PredDev &d = P->d;
        PCK(cudaMalloc(&d.param, P_NPARAM * 4));
        PCK(cudaMalloc(&d.m, P_NPARAM * 4));
        PCK(cudaMalloc(&d.v, P_NPARAM * 4));
        PCK(cudaMalloc(&d.grad, P_NPARAM * 4));
        PCK(cudaMalloc(&d.w1b, PH * 16 * 2));
        PCK(cudaMalloc(&d.w2b, PH * PH * 2));
        PCK(cudaMalloc(&d.ring, (size_t)P_RING * STAGE_BUCKETS * 4));
        PCK(cudaMalloc(&d.scores, STAGE_BUCKETS * 4));
        PCK(cudaMalloc(&d.act, (size_t)P_TRAIN * (PF + 2 * PH + 2) * 4));
        PCK(cudaMalloc(&d.state, 16));
        PCK(cudaMalloc(&d.loss, 8));
        PCK(cudaMalloc(&P->io, (size_t)P_TRAIN * 8 * 4));
    }
    ltpg_predictor_state *P = c->pred;
    std::vector<float> w;
    init_params(w, cfg->seed);
    PCK(cudaMemcpy(P->d.param, w.data(), P_NPARAM * 4, cudaMemcpyHostToDevice));
    PCK(cudaMemset(P->d.m, 0, P_NPARAM * 4));
    PCK(cudaMemset(P->d.v, 0, P_NPARAM * 4));
    PCK(cudaMemset(P->d.grad, 0, P_NPARAM * 4));
    PCK(cudaMemset(P->d.ring, 0, (size_t)P_RING * STAGE_BUCKETS * 4));
    PCK(cudaMemset(P->d.scores, 0, STAGE_BUCKETS * 4));
    PCK(cudaMemset(P->d.state, 0, 16));
    PCK(cudaMemset(P->d.loss, 0, 8));
    pred_cast<<<32, 256, 0, c->stream>>>(P->d);
    PCK(cudaGetLastError());
    P->lr = cfg->lr > 0.f ? cfg->lr : 3e-3f;
    P->train_every = cfg->train_every ? cfg->train_every : 1;
    P->steps_host = 0;
    c->pred_on = 1;
    c->pred_train = cfg->train != 0;
    c->stage_on = cfg->stage != 0;
    drop_graphs_ctx(c);
    return ltpg_sync(c);
}

int ltpg_predictor_stats(ltpg_ctx *c, float *loss, uint64_t *steps) {
    if (!c || !loss || !steps || !c->pred) return LTPG_ERR_STATE;
    uint32_t st[4];
    PCK(cudaMemcpyAsync(loss, c->pred->d.loss, 4, cudaMemcpyDeviceToHost, c->stream));
    PCK(cudaMemcpyAsync(st, c->pred->d.state, 16, cudaMemcpyDeviceToHost, c->stream));
    int r = ltpg_sync(c);
    if (r) return r;
    *steps = st[1];
    return LTPG_OK;
}

int ltpg_predictor_get_params(ltpg_ctx *c, float *host, size_t n) {
    if (!c || !host || !c->pred || n < (size_t)P_NPARAM) return LTPG_ERR_INVALID;
    PCK(cudaMemcpyAsync(host, c->pred->d.param, P_NPARAM * 4, cudaMemcpyDeviceToHost, c->stream));
    return ltpg_sync(c);
}

int ltpg_predictor_set_params(ltpg_ctx *c, const float *host, size_t n) {
    if (!c || !host || !c->pred || n < (size_t)P_NPARAM) return LTPG_ERR_INVALID;
    PCK(cudaMemcpyAsync(c->pred->d.param, host, P_NPARAM * 4, cudaMemcpyHostToDevice, c->stream));
    pred_cast<<<32, 256, 0, c->stream>>>(c->pred->d);
    PCK(cudaGetLastError());
    return ltpg_sync(c);
}

int ltpg_predictor_forward(ltpg_ctx *c, const float *host_x, uint32_t n, float *host_y) {
    if (!c || !host_x || !host_y || !c->pred || n == 0 || n > P_TRAIN) return LTPG_ERR_INVALID;
    ltpg_predictor_state *P = c->pred;
    PCK(cudaMemcpyAsync(P->io, host_x, (size_t)n * PF * 4, cudaMemcpyHostToDevice, c->stream));
    pred_forward<<<64, 256, 0, c->stream>>>(P->d, n, 2, P->io, P->io + P_TRAIN * PF);
    PCK(cudaGetLastError());
    PCK(cudaMemcpyAsync(host_y, P->io + P_TRAIN * PF, (size_t)n * 4, cudaMemcpyDeviceToHost, c->stream));
    return ltpg_sync(c);
}

int ltpg_predictor_gradients(ltpg_ctx *c, const float *host_x, const float *host_t, uint32_t n, float *host_grad) {
    if (!c || !host_x || !host_t || !host_grad || !c->pred || n == 0 || n > P_TRAIN) return LTPG_ERR_INVALID;
    ltpg_predictor_state *P = c->pred;
    // the training forward pass reads its samples from the ring; for a test we
    // run the given samples through the inference kernel and store the
    // activations with a host-side replay of mode 1's layout
    PCK(cudaMemcpyAsync(P->io, host_x, (size_t)n * PF * 4, cudaMemcpyHostToDevice, c->stream));
    pred_forward<<<64, 256, 0, c->stream>>>(P->d, n, 3, P->io, nullptr);
    PCK(cudaGetLastError());
    float *T = P->d.act + P_TRAIN * PF + 2 * P_TRAIN * PH + P_TRAIN;
    PCK(cudaMemcpyAsync(T, host_t, (size_t)n * 4, cudaMemcpyHostToDevice, c->stream));
    PCK(cudaMemsetAsync(P->d.grad, 0, P_NPARAM * 4, c->stream));
    pred_backward<<<64, 256, 0, c->stream>>>(P->d, n);
    PCK(cudaGetLastError());
    PCK(cudaMemcpyAsync(host_grad, P->d.grad, P_NPARAM * 4, cudaMemcpyDeviceToHost, c->stream));
    PCK(cudaMemsetAsync(P->d.grad, 0, P_NPARAM * 4, c->stream));
    PCK(cudaMemsetAsync(P->d.loss + 1, 0, 4, c->stream));
    return ltpg_sync(c);
}

}  // extern "C"

namespace ltpg {
// Enqueues one predictor step after a batch (also inside graph capture).
cudaError_t predictor_after_batch(ltpg_ctx *c) {
    ltpg_predictor_state *P = c->pred;
    if (!P || !c->pred_on) return cudaSuccess;
    // roll (and advance the ring), train, infer, select (and end the step)
    pred_roll<<<64, 256, 0, c->stream>>>(P->d, c->bucket_counts);
    count_launch(c);
    int trained = 0;
    if (c->pred_train) {
        pred_forward<<<P_TRAIN / 32, 64, 0, c->stream>>>(P->d, P_TRAIN, 1, nullptr, nullptr);
        pred_backward<<<128, 256, 0, c->stream>>>(P->d, P_TRAIN);
        pred_adam<<<18, 256, 0, c->stream>>>(P->d, P->lr, P_TRAIN);
        count_launch(c, 3);
        trained = 1;
    }
    pred_forward<<<STAGE_BUCKETS / 128, 256, 0, c->stream>>>(P->d, STAGE_BUCKETS, 0, nullptr, nullptr);
    count_launch(c);
    if (c->stage_on) {
        const uint32_t ways = c->launch_y.ways ? c->launch_y.ways : 4u;
        pred_select<<<SEL_BLOCKS, 1024, 0, c->stream>>>(P->d, STAGE_MAX_ENTRIES / ways, c->stage_bits,
                                                         c->stage_rank, c->stage_map, trained);
    } else {
        pred_step_done<<<1, 32, 0, c->stream>>>(P->d, trained);
    }
    count_launch(c);
    return cudaGetLastError();
}
}  // namespace ltpg

namespace ltpg {
void predictor_free(ltpg_ctx *c) {
    ltpg_predictor_state *P = c->pred;
    if (!P) return;
    for (void *ptr : {(void *)P->d.param, (void *)P->d.m, (void *)P->d.v, (void *)P->d.grad, (void *)P->d.w1b,
                      (void *)P->d.w2b, (void *)P->d.ring, (void *)P->d.scores, (void *)P->d.act,
                      (void *)P->d.state, (void *)P->d.loss, (void *)P->io})
        if (ptr) cudaFree(ptr);
    delete P;
    c->pred = nullptr;
}
}  // namespace ltpg
