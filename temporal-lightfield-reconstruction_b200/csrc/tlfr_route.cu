// tlfr_route.cu — learned routing (no counterpart in the reference: it is the
// addition that sends easy pixels to a fast path).  The fast path is the plain
// 1R pass that keeps the first surface when a second one opens instead of
// refetching at 2R (light_unit() in tlfr_query.cu), so the expensive full path
// runs only where the network is not confident.
//
//   features   eight cheap per-pixel features: depth, depth range and CoC
//              radius in the pixel, depth ranges within 3x3 and 5x5 tiles of
//              8x8 pixels (about the defocus radius), how much nearer the
//              nearest surface in that window is, motion magnitude, and a
//              coarse pass: the plain 1R pass on four of the pixel's output
//              samples, of which the fraction that needs the full path.
//   labels     1 when the fast path is as good as the plain method at the
//              pixel: within a tolerance of the plain pixel on every channel,
//              or, given the scene's ground truth, with a squared error against
//              it at most a tolerance above the plain pixel's (the plain method
//              and the fast path are both run on the frame).
//   network    8-64-64-1 MLP, ReLU, sigmoid output, binary cross-entropy.
//              Forward, backward and inference run on the tensor cores
//              (mma.sync m16n8k16, BF16 operands, FP32 accumulation); the
//              activations stay in registers between layers (the accumulator
//              tiles of one layer are the A operand tiles of the next).  Adam
//              updates FP32 master weights, which are then packed to BF16.
#include "tlfr_internal.h"

#include <cuda_bf16.h>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace tlfr
{

namespace
{

// ---------------------------------------------------------------------------
// features
// ---------------------------------------------------------------------------

// Per pixel over its input records ((y*W+x)*spp + k, 16 floats each:
// x, y, z/w, w, u, v, t, rgba, mv (3), dw/dx, dw/dy):
//   a = (log w min, log w max, CoC min, CoC max), b = (mean log w, max |motion|, hits, 0)
__global__ void k_feat_pixel(const float* __restrict__ rec, const int* __restrict__ hits, long long npix, int spp,
                             float c0, float c1, float4* __restrict__ fa, float4* __restrict__ fb)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x)
    {
        float lmin = 1e30f, lmax = -1e30f, cmin = 1e30f, cmax = -1e30f, lsum = 0, mmax = 0;
        for (int k = 0; k < spp; k++)
        {
            const float* r = rec + ((size_t)p * spp + k) * 16;
            const float w = fmaxf(r[3], 1e-6f);
            const float lw = logf(w);
            const float coc = c0 / w + c1;
            const float mx = r[11] / w, my = r[12] / w;
            lmin = fminf(lmin, lw);
            lmax = fmaxf(lmax, lw);
            cmin = fminf(cmin, coc);
            cmax = fmaxf(cmax, coc);
            lsum += lw;
            mmax = fmaxf(mmax, sqrtf(mx * mx + my * my));
        }
        fa[p] = make_float4(lmin, lmax, cmin, cmax);
        fb[p] = make_float4(lsum / (float)spp, mmax, (float)hits[p], 0.0f);
    }
}

// Coarse pass: 8x8-pixel tiles of (log w min, log w max, max |CoC|).
constexpr int kTile = 8;
__global__ void k_feat_tile(const float4* __restrict__ fa, int W, int H, int TW, int TH, float4* __restrict__ tiles)
{
    const int ntile = TW * TH;
    for (int ti = blockIdx.x * blockDim.x + threadIdx.x; ti < ntile; ti += gridDim.x * blockDim.x)
    {
        const int tx = ti % TW, ty = ti / TW;
        float lmin = 1e30f, lmax = -1e30f, cmax = 0;
        for (int y = ty * kTile; y < min(H, ty * kTile + kTile); y++)
            for (int x = tx * kTile; x < min(W, tx * kTile + kTile); x++)
            {
                const float4 a = fa[(long long)y * W + x];
                lmin = fminf(lmin, a.x);
                lmax = fmaxf(lmax, a.y);
                cmax = fmaxf(cmax, fmaxf(fabsf(a.z), fabsf(a.w)));
            }
        tiles[ti] = make_float4(lmin, lmax, cmax, 0.0f);
    }
}

// The eight features of each pixel (row-major [npix][8]):
//   0 mean log w            1 log w range in the pixel     2 max |CoC| in the pixel
//   3 mean log w minus the smallest log w within 5x5 tiles (a nearer surface that may blur over)
//   4 log w range within 3x3 tiles   5 log w range within 5x5 tiles
//   6 fraction of the pixel's probed output samples that the plain 1R pass sends to the full path
//   7 largest screen motion in the pixel
__global__ void k_feat_final(const float4* __restrict__ fa, const float4* __restrict__ fb,
                             const float4* __restrict__ tiles, const int* __restrict__ probe, int W, int H, int TW,
                             int TH, float* __restrict__ feats)
{
    const long long npix = (long long)W * H;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x)
    {
        const int x = (int)(p % W), y = (int)(p / W);
        const int tx = x / kTile, ty = y / kTile;
        const float4 a = fa[p], b = fb[p];
        float l3min = 1e30f, l3max = -1e30f, l5min = 1e30f, l5max = -1e30f, c5 = 0;
        for (int dy = -2; dy <= 2; dy++)
            for (int dx = -2; dx <= 2; dx++)
            {
                const int xx = tx + dx, yy = ty + dy;
                if (xx < 0 || yy < 0 || xx >= TW || yy >= TH)
                    continue;
                const float4 t = tiles[yy * TW + xx];
                l5min = fminf(l5min, t.x);
                l5max = fmaxf(l5max, t.y);
                c5 = fmaxf(c5, t.z);
                if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1)
                {
                    l3min = fminf(l3min, t.x);
                    l3max = fmaxf(l3max, t.y);
                }
            }
        float* f = feats + p * kRouteFeatures;
        f[0] = b.x;
        f[1] = a.y - a.x;
        f[2] = fmaxf(fabsf(a.z), fabsf(a.w));
        f[3] = b.x - l5min;
        f[4] = l3max - l3min;
        f[5] = l5max - l5min;
        f[6] = (float)probe[p] * (1.0f / kRouteProbes);
        f[7] = b.y;
    }
}

// Label 1 where the fast path is as good as the plain method: without a
// reference image, where it reproduces the plain pixel within tol on every
// channel; with one (the scene's ground truth), where its squared RGB error
// against the reference exceeds the plain pixel's by at most tol.
__global__ void k_labels(const float4* __restrict__ plain, const float4* __restrict__ fast,
                         const float4* __restrict__ ref, long long npix, float tol, float* __restrict__ labels)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x)
    {
        const float4 a = plain[p], b = fast[p];
        bool ok;
        if (ref)
        {
            const float4 r = ref[p];
            const float ea = (a.x - r.x) * (a.x - r.x) + (a.y - r.y) * (a.y - r.y) + (a.z - r.z) * (a.z - r.z);
            const float eb = (b.x - r.x) * (b.x - r.x) + (b.y - r.y) * (b.y - r.y) + (b.z - r.z) * (b.z - r.z);
            ok = eb <= ea + tol;
        }
        else
        {
            const float d = fmaxf(fmaxf(fabsf(a.x - b.x), fabsf(a.y - b.y)), fmaxf(fabsf(a.z - b.z), fabsf(a.w - b.w)));
            ok = d <= tol;
        }
        labels[p] = ok ? 1.0f : 0.0f;
    }
}

__global__ void k_route_flags(const float* __restrict__ prob, long long npix, float hi, unsigned char* __restrict__ fast)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npix; p += (long long)gridDim.x * blockDim.x)
        fast[p] = prob[p] > hi ? 1 : 0;
}

// ---------------------------------------------------------------------------
// network
// ---------------------------------------------------------------------------

constexpr int kF = kRouteFeatures;   // 8 inputs, padded to K = 16 for the first layer
constexpr int kK1 = 16;
constexpr int kH = 64;

// FP32 parameter block (row-major [out][in]); the trainable part is a prefix.
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kH * kK1;
constexpr int kOffW2 = kOffB1 + kH;
constexpr int kOffB2 = kOffW2 + kH * kH;
constexpr int kOffW3 = kOffB2 + kH;
constexpr int kOffB3 = kOffW3 + kH;
constexpr int kNumTrain = kOffB3 + 1;
constexpr int kOffMean = kNumTrain;               // input standardisation (fixed)
constexpr int kOffInvStd = kOffMean + kF;
constexpr int kNumParams = kOffInvStd + kF;

// BF16 operand block: the B operands (16 x 8) of every mma, fragment by fragment
// as the lanes hold them: lane (g, t) of fragment f has elements (k, n) = (2t, g),
// (2t + 1, g), (2t + 8, g), (2t + 9, g) in 8 bytes at (f * 32 + lane).  A fragment
// is then one coalesced 64-bit load, two L1 wavefronts; read from the row-major
// matrices it took two loads of eight each, which bound inference (2.07 M rows:
// 329 us, now 135).
// Fragments: layer 1 by output tile; layer 2 by (output tile, k tile), W2 and then
// its transpose; layer 3, padded to 8 outputs, by k tile.
constexpr int kFragW1 = 0;
constexpr int kFragW2 = kFragW1 + 8;
constexpr int kFragW2T = kFragW2 + 32;
constexpr int kFragW3 = kFragW2T + 32;
constexpr int kNumHalf = (kFragW3 + 4) * 128;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    uint32_t u;
    memcpy(&u, &v, 4);
    return u;
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// D += A * B, m16n8k16, BF16 operands, FP32 accumulators.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// This lane's part of B fragment f.
__device__ __forceinline__ void load_b(const __nv_bfloat16* w, int f, uint32_t& b0, uint32_t& b1)
{
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(w) + f * 32 + (threadIdx.x & 31));
    b0 = v.x;
    b1 = v.y;
}

// Accumulator tiles c[2kk], c[2kk+1] (16 x 8 each) as the A operand of k-tile kk.
__device__ __forceinline__ void acc_to_a(const float (&c0)[4], const float (&c1)[4], uint32_t (&a)[4])
{
    a[0] = pack_bf16(c0[0], c0[1]);
    a[1] = pack_bf16(c0[2], c0[3]);
    a[2] = pack_bf16(c1[0], c1[1]);
    a[3] = pack_bf16(c1[2], c1[3]);
}

// Forward pass of one 16-row tile.  Lane (g = lane/4, t = lane%4) holds rows
// g and g + 8, whose features are at row[0] and row[1] (zero where not valid).
// Outputs: h1, h2 after ReLU, rounded to BF16 (the values the next layer
// multiplies), columns 8j + 2t (+1); logits y for rows g and g+8 (valid on lanes
// with t == 0).  PAIRS: the features start on 8 bytes, and two are
// loaded at a time (feature_pairs()).
struct Tile
{
    float h1[8][4], h2[8][4];
    uint32_t x[4];
    float y0, y8;
};

template <bool PAIRS>
__device__ __forceinline__ void tile_forward(const float* __restrict__ P, const __nv_bfloat16* __restrict__ Wh,
                                             const float* __restrict__ feats, const int (&row)[2], const bool (&valid)[2],
                                             Tile& T)
{
    const int t = threadIdx.x & 3;
    float xv[2][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
    {
        float2 f = make_float2(0, 0);
        if (valid[h])
        {
            const float* p = feats + (size_t)row[h] * kF + 2 * t;
            f = PAIRS ? *reinterpret_cast<const float2*>(p) : make_float2(p[0], p[1]);
        }
        const int col = 2 * t;
        xv[h][0] = valid[h] ? (f.x - P[kOffMean + col]) * P[kOffInvStd + col] : 0.0f;
        xv[h][1] = valid[h] ? (f.y - P[kOffMean + col + 1]) * P[kOffInvStd + col + 1] : 0.0f;
    }
    T.x[0] = pack_bf16(xv[0][0], xv[0][1]);
    T.x[1] = pack_bf16(xv[1][0], xv[1][1]);
    T.x[2] = 0;
    T.x[3] = 0;
    // layer 1
#pragma unroll
    for (int j = 0; j < 8; j++)
    {
        float c[4] = { 0, 0, 0, 0 };
        uint32_t b0, b1;
        load_b(Wh, kFragW1 + j, b0, b1);
        mma16816(c, T.x, b0, b1);
        const float2 bias = *reinterpret_cast<const float2*>(P + kOffB1 + 8 * j + 2 * t);
#pragma unroll
        for (int q = 0; q < 4; q++)
            T.h1[j][q] = bf16_round(fmaxf(c[q] + (q & 1 ? bias.y : bias.x), 0.0f));
    }
    // layer 2
    uint32_t a[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
        acc_to_a(T.h1[2 * kk], T.h1[2 * kk + 1], a[kk]);
#pragma unroll
    for (int j = 0; j < 8; j++)
    {
        float c[4] = { 0, 0, 0, 0 };
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
        {
            uint32_t b0, b1;
            load_b(Wh, kFragW2 + 4 * j + kk, b0, b1);
            mma16816(c, a[kk], b0, b1);
        }
        const float2 bias = *reinterpret_cast<const float2*>(P + kOffB2 + 8 * j + 2 * t);
#pragma unroll
        for (int q = 0; q < 4; q++)
            T.h2[j][q] = bf16_round(fmaxf(c[q] + (q & 1 ? bias.y : bias.x), 0.0f));
    }
    // layer 3 (one output column of an 8-wide tile)
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
        acc_to_a(T.h2[2 * kk], T.h2[2 * kk + 1], a[kk]);
    float c[4] = { 0, 0, 0, 0 };
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
    {
        uint32_t b0, b1;
        load_b(Wh, kFragW3 + kk, b0, b1);
        mma16816(c, a[kk], b0, b1);
    }
    T.y0 = c[0] + P[kOffB3];
    T.y8 = c[2] + P[kOffB3];
}

__device__ __forceinline__ float sigmoid(float y) { return 1.0f / (1.0f + expf(-y)); }

// Inference: probability that each pixel is a single surface.
template <bool PAIRS>
__global__ void __launch_bounds__(128) k_mlp_infer(const float* __restrict__ P, const __nv_bfloat16* __restrict__ Wh,
                                                    const float* __restrict__ feats, long long n, float* __restrict__ prob)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long tile = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile * 16 < n; tile += warps)
    {
        const long long r0 = tile * 16;
        const int nrows = (int)min(16LL, n - r0);
        const int row[2] = { (int)(r0 + g), (int)(r0 + g + 8) };
        const bool valid[2] = { g < nrows, g + 8 < nrows };
        Tile T;
        tile_forward<PAIRS>(P, Wh, feats, row, valid, T);
        if (t == 0)
        {
            if (g < nrows)
                prob[r0 + g] = sigmoid(T.y0);
            if (g + 8 < nrows)
                prob[r0 + g + 8] = sigmoid(T.y8);
        }
    }
}

// Row index of the k-th example of a training step's minibatch.
__device__ __forceinline__ int batch_row(unsigned seed, unsigned step, unsigned k, unsigned n)
{
    unsigned h = k * 0x9e3779b1u ^ (step * 0x85ebca6bu + seed);
    h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; h ^= h >> 16;
    return (int)(h % n);
}

// Sum over the 8 row groups (lanes with the same t) of a per-lane value.
__device__ __forceinline__ float sum_groups(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

constexpr int kTrainWarps = 4;
constexpr int kTrainGroups = 8;

// Forward + backward of binary cross-entropy (mean over the batch) for a
// minibatch; gradients are added into grad (FP32, kNumTrain).  Rows are the
// minibatch rows: row k = batch_row(seed, step, k, n), or k itself when
// all_rows is set (the gradient over exactly rows 0..batch-1).
// A block takes kTrainWarps tiles of 16 rows at a time: each warp runs one tile
// forward and back and stages what the weight gradients contract over the rows;
// then warp w accumulates rows 16w..16w+15 of dL/dW2 and dL/dW1 over the block's
// tiles in its mma accumulators.  (Adding every tile's products to shared memory
// with float atomics took 544 us for 262144 rows; this 169 us, 121 with the weights
// read as fragments.)  The mma truncates, so the error grows with the number of them
// that an accumulator goes through: after kTrainGroups groups the sums move to
// shared memory.  Relative error of the gradient of 4194304 rows against the BF16
// network in 64 bits: 6.4e-7; 2.9e-6 without this, 6.3e-7 with atomics per tile.
template <bool PAIRS>
__global__ void __launch_bounds__(kTrainWarps * 32)
k_mlp_train(const float* __restrict__ P, const __nv_bfloat16* __restrict__ Wh, const float* __restrict__ feats,
            const float* __restrict__ labels, int n, int batch, unsigned seed, unsigned step, int all_rows,
            float* __restrict__ grad, float* __restrict__ loss_out)
{
    static_assert(kTrainWarps * 16 == kH, "a warp owns 16 rows of the weight gradients");
    __shared__ float s_grad[kNumTrain];
    // written two values at a time
    __shared__ alignas(4) __nv_bfloat16 s_h1[kTrainWarps][16][kH];
    __shared__ alignas(4) __nv_bfloat16 s_dh2[kTrainWarps][16][kH];
    __shared__ alignas(4) __nv_bfloat16 s_dh1[kTrainWarps][16][kH];
    __shared__ alignas(4) __nv_bfloat16 s_x[kTrainWarps][16][kF];
    __shared__ float s_loss;
    for (int i = threadIdx.x; i < kNumTrain; i += blockDim.x)
        s_grad[i] = 0.0f;
    if (threadIdx.x == 0)
        s_loss = 0.0f;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float inv_batch = 1.0f / (float)batch;
    float loss = 0.0f;
    float c2[8][4] = {}, c1[4] = {};        // this warp's rows of dL/dW2 and dL/dW1, over the last groups
    int groups = 0;
    float gw3[8][2] = {}, gb2[8][2] = {}, gb1[8][2] = {}, gb3 = 0.0f;     // this lane's rows' sums
    for (long long first = (long long)blockIdx.x * kTrainWarps * 16; first < batch;
         first += (long long)gridDim.x * kTrainWarps * 16)
    {
        const long long k0 = first + warp * 16;
        const int nrows = (int)max(0LL, min(16LL, batch - k0));
        const bool valid[2] = { g < nrows, g + 8 < nrows };
        int row[2];
        for (int h = 0; h < 2; h++)
        {
            const int k = valid[h] ? (int)(k0 + g + 8 * h) : 0;
            row[h] = all_rows ? k : batch_row(seed, step, (unsigned)k, (unsigned)n);
        }
        Tile T;
        tile_forward<PAIRS>(P, Wh, feats, row, valid, T);
        // dL/dy = (p - label) / batch for rows g and g + 8, broadcast to the lane group
        float dy0 = 0.0f, dy8 = 0.0f;
        if (t == 0)
        {
            if (valid[0])
            {
                const float p = sigmoid(T.y0), lab = labels[row[0]];
                dy0 = (p - lab) * inv_batch;
                loss -= (lab * logf(fmaxf(p, 1e-7f)) + (1 - lab) * logf(fmaxf(1 - p, 1e-7f))) * inv_batch;
            }
            if (valid[1])
            {
                const float p = sigmoid(T.y8), lab = labels[row[1]];
                dy8 = (p - lab) * inv_batch;
                loss -= (lab * logf(fmaxf(p, 1e-7f)) + (1 - lab) * logf(fmaxf(1 - p, 1e-7f))) * inv_batch;
            }
            gb3 += dy0 + dy8;
        }
        dy0 = __shfl_sync(0xffffffffu, dy0, lane & ~3);
        dy8 = __shfl_sync(0xffffffffu, dy8, lane & ~3);
        // layer 3: grad w3, b3; dh2 = dy * w3 * relu'(h2)
        float dh2[8][4];
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
            for (int q = 0; q < 2; q++)
            {
                const int col = 8 * j + 2 * t + q;
                const float w3 = bf16_round(P[kOffW3 + col]);
                gw3[j][q] += dy0 * T.h2[j][q] + dy8 * T.h2[j][q + 2];
                dh2[j][q] = T.h2[j][q] > 0.0f ? bf16_round(dy0 * w3) : 0.0f;
                dh2[j][q + 2] = T.h2[j][q + 2] > 0.0f ? bf16_round(dy8 * w3) : 0.0f;
                gb2[j][q] += dh2[j][q] + dh2[j][q + 2];
            }
        // dh1 = dh2 * W2 (row-major [n][k]; the B operand is W2 transposed) * relu'(h1)
        uint32_t a[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
            acc_to_a(dh2[2 * kk], dh2[2 * kk + 1], a[kk]);
        __syncthreads();        // the previous group's staged tiles have been read
#pragma unroll
        for (int j = 0; j < 8; j++)
        {
            float c[4] = { 0, 0, 0, 0 };
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
            {
                uint32_t b0, b1;
                load_b(Wh, kFragW2T + 4 * j + kk, b0, b1);
                mma16816(c, a[kk], b0, b1);
            }
            float dh1[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
                dh1[q] = T.h1[j][q] > 0.0f ? bf16_round(c[q]) : 0.0f;
#pragma unroll
            for (int q = 0; q < 2; q++)
                gb1[j][q] += dh1[q] + dh1[q + 2];
            // stage h1, dh2, dh1 (row-major [row][col]) for the weight gradients,
            // which contract over the rows
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                const int r = g + 8 * h, col = 8 * j + 2 * t;
                *reinterpret_cast<uint32_t*>(&s_h1[warp][r][col]) = pack_bf16(T.h1[j][2 * h], T.h1[j][2 * h + 1]);
                *reinterpret_cast<uint32_t*>(&s_dh2[warp][r][col]) = pack_bf16(dh2[j][2 * h], dh2[j][2 * h + 1]);
                *reinterpret_cast<uint32_t*>(&s_dh1[warp][r][col]) = pack_bf16(dh1[2 * h], dh1[2 * h + 1]);
            }
        }
        *reinterpret_cast<uint32_t*>(&s_x[warp][g][2 * t]) = T.x[0];
        *reinterpret_cast<uint32_t*>(&s_x[warp][g + 8][2 * t]) = T.x[1];
        __syncthreads();
        // grad W2[n][k] = sum_rows dh2[row][n] * h1[row][k]; grad W1[n][k] = sum_rows dh1[row][n] * x[row][k].
        // A = (dh)^T tile [n][row] (16 x 16), B = (h1 or x) as (k = row, n = col).
        auto at = [&](const __nv_bfloat16* m, int ld, int r, int c) {
            return (uint32_t)reinterpret_cast<const uint16_t&>(m[r * ld + c]) |
                   ((uint32_t)reinterpret_cast<const uint16_t&>(m[(r + 1) * ld + c]) << 16);
        };
        for (int rt = 0; rt < kTrainWarps; rt++)
        {
            uint32_t A2[4], A1[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const int nn = 16 * warp + g + 8 * (q & 1);
                const int rr = 2 * t + 8 * (q >> 1);
                A2[q] = at(&s_dh2[rt][0][0], kH, rr, nn);
                A1[q] = at(&s_dh1[rt][0][0], kH, rr, nn);
            }
#pragma unroll
            for (int j = 0; j < 8; j++)
            {
                const int kc = 8 * j + g;
                mma16816(c2[j], A2, at(&s_h1[rt][0][0], kH, 2 * t, kc), at(&s_h1[rt][0][0], kH, 2 * t + 8, kc));
            }
            // x columns 0..7
            mma16816(c1, A1, at(&s_x[rt][0][0], kF, 2 * t, g), at(&s_x[rt][0][0], kF, 2 * t + 8, g));
        }
        // the weight gradients' sums, each element held by one lane of the block
        if (++groups % kTrainGroups == 0 || first + (long long)gridDim.x * kTrainWarps * 16 >= batch)
        {
            const bool more = groups > kTrainGroups;
            auto add = [more](float& sum, float& c) {
                sum = more ? sum + c : c;
                c = 0.0f;
            };
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const int nn = 16 * warp + g + 8 * (q >> 1);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    add(s_grad[kOffW2 + nn * kH + 8 * j + 2 * t + (q & 1)], c2[j][q]);
                add(s_grad[kOffW1 + nn * kK1 + 2 * t + (q & 1)], c1[q]);
            }
        }
    }
    // the others, summed over the block's warps
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int q = 0; q < 2; q++)
        {
            const float w3 = sum_groups(gw3[j][q]), b2 = sum_groups(gb2[j][q]), b1 = sum_groups(gb1[j][q]);
            if (g == 0)
            {
                const int col = 8 * j + 2 * t + q;
                atomicAdd(&s_grad[kOffW3 + col], w3);
                atomicAdd(&s_grad[kOffB2 + col], b2);
                atomicAdd(&s_grad[kOffB1 + col], b1);
            }
        }
    gb3 = sum_groups(gb3);
    loss = sum_groups(loss);
    if (lane == 0)
    {
        atomicAdd(&s_grad[kOffB3], gb3);
        atomicAdd(&s_loss, loss);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kNumTrain; i += blockDim.x)
        if (s_grad[i] != 0.0f)
            atomicAdd(&grad[i], s_grad[i]);
    if (threadIdx.x == 0 && loss_out)
        atomicAdd(loss_out, s_loss);
}

// Adam on the FP32 master weights; clears the gradient for the next step.
__global__ void k_adam(float* __restrict__ P, float* __restrict__ grad, float* __restrict__ m, float* __restrict__ v,
                       float lr, float b1, float b2, float eps, float bc1, float bc2)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNumTrain; i += gridDim.x * blockDim.x)
    {
        const float gi = grad[i];
        const float mi = b1 * m[i] + (1 - b1) * gi;
        const float vi = b2 * v[i] + (1 - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        P[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
        grad[i] = 0.0f;
    }
}

// BF16 operand block from the FP32 master weights.
__global__ void k_pack(const float* __restrict__ P, __nv_bfloat16* __restrict__ Wh)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNumHalf; i += gridDim.x * blockDim.x)
    {
        const int f = i >> 7, lane = (i >> 2) & 31;
        const int n = lane >> 2, k = 2 * (lane & 3) + (i & 1) + 8 * ((i >> 1) & 1);
        float v;
        if (f < kFragW2)
            v = P[kOffW1 + (8 * f + n) * kK1 + k];
        else if (f < kFragW2T)
            v = P[kOffW2 + (8 * ((f - kFragW2) >> 2) + n) * kH + 16 * ((f - kFragW2) & 3) + k];
        else if (f < kFragW3)
            v = P[kOffW2 + (16 * ((f - kFragW2T) & 3) + k) * kH + 8 * ((f - kFragW2T) >> 2) + n];
        else
            v = n == 0 ? P[kOffW3 + 16 * (f - kFragW3) + k] : 0.0f;
        Wh[i] = __float2bfloat16_rn(v);
    }
}

} // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

#define CKR(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) { err = std::string(#x) + ": " + cudaGetErrorString(_e); return (_e == cudaErrorMemoryAllocation) ? TLFR_OOM : TLFR_CUDA; } } while (0)

int route_num_params() { return kNumParams; }
int route_num_trainable() { return kNumTrain; }

tlfr_status route_alloc(Route& r, std::string& err)
{
    CKR(cudaDeviceGetAttribute(&r.num_sms, cudaDevAttrMultiProcessorCount, r.device));
    CKR(cudaMalloc(&r.params, sizeof(float) * kNumParams));
    CKR(cudaMalloc(&r.grad, sizeof(float) * kNumTrain));
    CKR(cudaMalloc(&r.m, sizeof(float) * kNumTrain));
    CKR(cudaMalloc(&r.v, sizeof(float) * kNumTrain));
    CKR(cudaMalloc(&r.half, sizeof(__nv_bfloat16) * kNumHalf));
    CKR(cudaMalloc(&r.loss, sizeof(float)));
    CKR(cudaMemset(r.grad, 0, sizeof(float) * kNumTrain));
    CKR(cudaMemset(r.m, 0, sizeof(float) * kNumTrain));
    CKR(cudaMemset(r.v, 0, sizeof(float) * kNumTrain));
    return TLFR_OK;
}

void route_free(Route& r)
{
    void* p[] = { r.params, r.grad, r.m, r.v, r.half, r.loss };
    for (void* q : p)
        if (q) cudaFree(q);
    r = Route{};
}

// He-style initialisation from a fixed seed; standardisation from the caller.
tlfr_status route_init(Route& r, unsigned seed, const float* mean, const float* inv_std, cudaStream_t s, std::string& err)
{
    std::vector<float> h(kNumParams, 0.0f);
    uint32_t st = seed * 747796405u + 2891336453u;
    auto rnd = [&]() {   // uniform in [-1, 1)
        st = st * 747796405u + 2891336453u;
        uint32_t w = ((st >> ((st >> 28u) + 4u)) ^ st) * 277803737u;
        w = (w >> 22u) ^ w;
        return (float)w / 2147483648.0f - 1.0f;
    };
    const float s1 = sqrtf(6.0f / kF), s2 = sqrtf(6.0f / kH), s3 = sqrtf(3.0f / kH);
    for (int n = 0; n < kH; n++)
        for (int k = 0; k < kF; k++)
            h[kOffW1 + n * kK1 + k] = s1 * rnd();
    for (int i = 0; i < kH * kH; i++)
        h[kOffW2 + i] = s2 * rnd();
    for (int i = 0; i < kH; i++)
        h[kOffW3 + i] = s3 * rnd();
    for (int k = 0; k < kF; k++)
    {
        h[kOffMean + k] = mean ? mean[k] : 0.0f;
        h[kOffInvStd + k] = inv_std ? inv_std[k] : 1.0f;
    }
    r.step = 0;
    CKR(cudaMemcpyAsync(r.params, h.data(), sizeof(float) * kNumParams, cudaMemcpyHostToDevice, s));
    CKR(cudaMemsetAsync(r.m, 0, sizeof(float) * kNumTrain, s));
    CKR(cudaMemsetAsync(r.v, 0, sizeof(float) * kNumTrain, s));
    CKR(cudaMemsetAsync(r.grad, 0, sizeof(float) * kNumTrain, s));
    k_pack<<<(kNumHalf + 255) / 256, 256, 0, s>>>(r.params, r.half);
    CKR(cudaStreamSynchronize(s));
    return TLFR_OK;
}

tlfr_status route_set_params(Route& r, const float* host_params, cudaStream_t s, std::string& err)
{
    CKR(cudaMemcpyAsync(r.params, host_params, sizeof(float) * kNumParams, cudaMemcpyHostToDevice, s));
    k_pack<<<(kNumHalf + 255) / 256, 256, 0, s>>>(r.params, r.half);
    CKR(cudaStreamSynchronize(s));
    return TLFR_OK;
}

tlfr_status route_get_params(Route& r, float* host_params, cudaStream_t s, std::string& err)
{
    CKR(cudaMemcpyAsync(host_params, r.params, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost, s));
    CKR(cudaStreamSynchronize(s));
    return TLFR_OK;
}

// The caller's features may start at any float.  A row is 32 bytes, so all pairs
// lie alike, and the kernels have a form for each case (looking at the pointer in
// the kernel: 1080p inference and the gradient of 262144 rows 312 us against 302).
static bool feature_pairs(const float* d_feats) { return (reinterpret_cast<size_t>(d_feats) & 7) == 0; }

static int train_blocks(const Route& r, int batch)
{
    return std::max(1, std::min(r.num_sms * 4, (batch + 16 * kTrainWarps - 1) / (16 * kTrainWarps)));
}

tlfr_status route_gradient(Route& r, const float* d_feats, const float* d_labels, int n, float* host_grad,
                           float* host_loss, cudaStream_t s, std::string& err)
{
    CKR(cudaMemsetAsync(r.grad, 0, sizeof(float) * kNumTrain, s));
    CKR(cudaMemsetAsync(r.loss, 0, sizeof(float), s));
    const auto kernel = feature_pairs(d_feats) ? k_mlp_train<true> : k_mlp_train<false>;
    kernel<<<train_blocks(r, n), kTrainWarps * 32, 0, s>>>(r.params, r.half, d_feats, d_labels, n, n, 0, 0, 1, r.grad,
                                                          r.loss);
    CKR(cudaGetLastError());
    CKR(cudaMemcpyAsync(host_grad, r.grad, sizeof(float) * kNumTrain, cudaMemcpyDeviceToHost, s));
    if (host_loss)
        CKR(cudaMemcpyAsync(host_loss, r.loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    CKR(cudaStreamSynchronize(s));
    CKR(cudaMemsetAsync(r.grad, 0, sizeof(float) * kNumTrain, s));
    return TLFR_OK;
}

tlfr_status route_train(Route& r, const float* d_feats, const float* d_labels, int n, int steps, int batch, float lr,
                        unsigned seed, float* host_loss, cudaStream_t s, std::string& err)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const auto kernel = feature_pairs(d_feats) ? k_mlp_train<true> : k_mlp_train<false>;
    CKR(cudaMemsetAsync(r.loss, 0, sizeof(float), s));
    for (int k = 0; k < steps; k++)
    {
        r.step++;
        const bool last = k == steps - 1;
        if (last)
            CKR(cudaMemsetAsync(r.loss, 0, sizeof(float), s));
        kernel<<<train_blocks(r, batch), kTrainWarps * 32, 0, s>>>(r.params, r.half, d_feats, d_labels, n, batch, seed,
                                                                  (unsigned)r.step, 0, r.grad, r.loss);
        k_adam<<<(kNumTrain + 255) / 256, 256, 0, s>>>(r.params, r.grad, r.m, r.v, lr, b1, b2, eps,
                                                       1.0f - powf(b1, (float)r.step), 1.0f - powf(b2, (float)r.step));
        k_pack<<<(kNumHalf + 255) / 256, 256, 0, s>>>(r.params, r.half);
    }
    CKR(cudaGetLastError());
    if (host_loss)
        CKR(cudaMemcpyAsync(host_loss, r.loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    CKR(cudaStreamSynchronize(s));
    return TLFR_OK;
}

tlfr_status route_predict(Route& r, const float* d_feats, long long n, float* d_prob, cudaStream_t s, std::string& err)
{
    const long long tiles = (n + 15) / 16;
    const int blocks = (int)std::max(1LL, std::min((long long)r.num_sms * 8, (tiles + 3) / 4));
    const auto kernel = feature_pairs(d_feats) ? k_mlp_infer<true> : k_mlp_infer<false>;
    kernel<<<blocks, 128, 0, s>>>(r.params, r.half, d_feats, n, d_prob);
    CKR(cudaGetLastError());
    return TLFR_OK;
}

tlfr_status route_features(Ctx& c, float* d_feats, std::string& err)
{
    const long long npix = (long long)c.W * c.H;
    const int TW = (c.W + kTile - 1) / kTile, TH = (c.H + kTile - 1) / kTile;
    if (!c.route_fa)
    {
        CKR(cudaMalloc(&c.route_fa, sizeof(float4) * (2 * npix + (size_t)TW * TH) + sizeof(int) * npix));
    }
    float4* fa = c.route_fa;
    float4* fb = c.route_fa + npix;
    float4* tiles = c.route_fa + 2 * npix;
    int* probe = reinterpret_cast<int*>(c.route_fa + 2 * npix + (size_t)TW * TH);
    const int blocks = (int)std::max(1LL, std::min((long long)c.num_sms * 16, (npix + 255) / 256));
    k_feat_pixel<<<blocks, 256, 0, c.stream>>>(c.cur_records, c.hits, npix, c.spp_in, c.coc[0], c.coc[1], fa, fb);
    k_feat_tile<<<(TW * TH + 127) / 128, 128, 0, c.stream>>>(fa, c.W, c.H, TW, TH, tiles);
    const tlfr_status ps = route_probe(c, probe);
    if (ps != TLFR_OK)
    {
        err = c.error;
        return ps;
    }
    k_feat_final<<<blocks, 256, 0, c.stream>>>(fa, fb, tiles, probe, c.W, c.H, TW, TH, d_feats);
    c.launches += 3;
    CKR(cudaGetLastError());
    return TLFR_OK;
}

tlfr_status route_labels_from(Ctx& c, const float4* d_plain, const float4* d_fast, const float4* d_ref, float tol,
                              float* d_labels, std::string& err)
{
    const long long npix = (long long)c.W * c.H;
    const int blocks = (int)std::max(1LL, std::min((long long)c.num_sms * 16, (npix + 255) / 256));
    k_labels<<<blocks, 256, 0, c.stream>>>(d_plain, d_fast, d_ref, npix, tol, d_labels);
    c.launches++;
    CKR(cudaGetLastError());
    return TLFR_OK;
}

tlfr_status route_flags(Ctx& c, const float* d_prob, float hi, unsigned char* d_fast, std::string& err)
{
    const long long npix = (long long)c.W * c.H;
    const int blocks = (int)std::max(1LL, std::min((long long)c.num_sms * 16, (npix + 255) / 256));
    k_route_flags<<<blocks, 256, 0, c.stream>>>(d_prob, npix, hi, d_fast);
    c.launches++;
    CKR(cudaGetLastError());
    return TLFR_OK;
}

} // namespace tlfr
