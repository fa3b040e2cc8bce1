// Subtree-size model for the learned schedule: a 16-64-64-1 perceptron with
// ReLU hidden layers, FP16 weights and inputs, FP32 accumulation, trained on
// the GPU by the kernels below (forward, gradient, Adam).  Target: log1p of a
// root task's search-tree nodes.  The model only orders the roots (largest
// predicted first); it never prunes, so the result set does not depend on it.
//
// Parameter layout (FP32 master copy and FP16 working copy alike):
//   W1[64][16] b1[64] W2[64][64] b2[64] W3[64] b3
// Features per root x (root_features_kernel), each log1p-scaled:
//   0 k, 1 depth (0 for a root task), 2 deg x, 3 |V| - deg x,
//   4 candidate U count (ids > x), 5 exclusion count (ids < x),
//   6 sum deg y over N(x) (2-hop size with repeats), 7 max deg y, 8 min deg y,
//   9 mean deg y, 10 |V|, 11 |U|, 12 sum over y of |N(y) above x|,
//   13 sum over y of |N(y) below x|, 14 #y with deg y <= k + 1,
//   15 log2 bucket of deg x.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "enum_core.cuh"

namespace gmk {
namespace mlp {

constexpr int F = 16;
constexpr int H = 64;
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + H * F;
constexpr int OFF_W2 = OFF_B1 + H;
constexpr int OFF_B2 = OFF_W2 + H * H;
constexpr int OFF_W3 = OFF_B2 + H;
constexpr int OFF_B3 = OFF_W3 + H;
constexpr int NP = OFF_B3 + 1;   // 5313 parameters

// One warp per root: the 16 features of root task x.
__global__ void root_features_kernel(GraphView g, uint32_t k, __half* out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t x = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (x >= g.nl) return;
    const uint32_t d = degree(g, (uint32_t)x);
    const uint32_t* row = g.adj + g.off[x];
    unsigned long long sum = 0, above = 0, below = 0, small = 0, words = 0;
    uint32_t mx = 0, mn = 0xFFFFFFFFu;
    for (uint32_t i = lane; i < d; i += 32) {
        const uint32_t y = row[i];
        const uint32_t dy = degree(g, y);
        sum += dy;
        mx = dy > mx ? dy : mx;
        mn = dy < mn ? dy : mn;
        small += dy <= k + 1 ? 1u : 0u;
        const uint32_t a = count_above(g, y, (uint32_t)x, &words);
        above += a;
        below += dy - a - 1;   // y's neighbours below x (x itself excluded)
    }
    for (int o = 16; o; o >>= 1) {
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        above += __shfl_xor_sync(0xFFFFFFFFu, above, o);
        below += __shfl_xor_sync(0xFFFFFFFFu, below, o);
        small += __shfl_xor_sync(0xFFFFFFFFu, small, o);
        const uint32_t a = __shfl_xor_sync(0xFFFFFFFFu, mx, o);
        const uint32_t b = __shfl_xor_sync(0xFFFFFFFFu, mn, o);
        mx = a > mx ? a : mx;
        mn = b < mn ? b : mn;
    }
    if (lane != 0) return;
    const uint32_t nv = g.n - g.nl;
    float f[F];
    f[0] = (float)k;
    f[1] = 0.f;
    f[2] = (float)d;
    f[3] = (float)(nv - d);
    f[4] = (float)(g.nl - 1 - x);
    f[5] = (float)x;
    f[6] = (float)sum;
    f[7] = (float)mx;
    f[8] = d ? (float)mn : 0.f;
    f[9] = d ? (float)sum / (float)d : 0.f;
    f[10] = (float)nv;
    f[11] = (float)g.nl;
    f[12] = (float)above;
    f[13] = (float)below;
    f[14] = (float)small;
    f[15] = (float)(32 - __clz(d | 1u));
    for (int i = 0; i < F; ++i) out[x * F + i] = __float2half_rn(log1pf(f[i]));
}

// Samples go through the model in tiles of kTile, one tile per block at a time;
// the block's 16 x 16 threads each own 4 x 4 outputs of every 64 x 64 product
// (FP32 multiply-adds in the order of a plain loop over k).  Operands are in
// shared memory with k as the slow index, so that a k step reads one float4 per
// operand and thread.  Rows are padded by 4 words: a transposed store then
// spreads over the banks, and float4 reads stay aligned.
constexpr int kTile = 64;
constexpr int kThreads = 256;
constexpr int kPitch = kTile + 4;

struct TileShared {
    float w1t[F][kPitch];        // W1 transposed: [f][j]
    float w2t[H][kPitch];        // W2 transposed: [q][j]
    float b1[H], b2[H], w3[H];
    float xt[F][kPitch];         // [f][sample]
    float h1t[H][kPitch];        // [q][sample]
    float h2t[H][kPitch];        // [j][sample]; the backward pass: dh2 likewise
    float out[kTile];
    float b3;
};
// What only the backward pass keeps.
struct TileGrad {
    float w2[H][kPitch];         // [j][q]
    float x[kTile][F + 4];       // [sample][f]
    float h1[kTile][kPitch];     // [sample][q]; later dh1
    float dh2[kTile][kPitch];    // [sample][j]
    float dout[kTile];
    float red[kThreads];
};

__device__ __forceinline__ void load_weights(const __half* w, TileShared& s) {
    for (int i = threadIdx.x; i < H * F; i += kThreads) s.w1t[i % F][i / F] = __half2float(w[OFF_W1 + i]);
    for (int i = threadIdx.x; i < H * H; i += kThreads) s.w2t[i % H][i / H] = __half2float(w[OFF_W2 + i]);
    for (int i = threadIdx.x; i < H; i += kThreads) {
        s.b1[i] = __half2float(w[OFF_B1 + i]);
        s.b2[i] = __half2float(w[OFF_B2 + i]);
        s.w3[i] = __half2float(w[OFF_W3 + i]);
    }
    if (threadIdx.x == 0) s.b3 = __half2float(w[OFF_B3]);
}

// acc[a][b] += sum over k of left[k][4 ty + a] * right[k][4 tx + b]
template <int K, int PL, int PR>
__device__ __forceinline__ void product(const float (*left)[PL], const float (*right)[PR], int ty, int tx,
                                        float (&acc)[4][4]) {
    #pragma unroll 8
    for (int k = 0; k < K; ++k) {
        const float4 l = *reinterpret_cast<const float4*>(&left[k][4 * ty]);
        const float4 r = *reinterpret_cast<const float4*>(&right[k][4 * tx]);
        const float la[4] = {l.x, l.y, l.z, l.w}, ra[4] = {r.x, r.y, r.z, r.w};
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
            #pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(la[a], ra[b], acc[a][b]);
        }
    }
}

// The same where an operand may be infinite or NaN: a term whose left factor (kBoth:
// either factor) is zero is left out, as a unit that is off contributes nothing.
template <int K, bool kBoth, int PL, int PR>
__device__ __forceinline__ void product_of_nonzeros(const float (*left)[PL], const float (*right)[PR], int ty,
                                                 int tx, float (&acc)[4][4]) {
    #pragma unroll 1
    for (int k = 0; k < K; ++k) {
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
            #pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float l = left[k][4 * ty + a], r = right[k][4 * tx + b];
                if (l != 0.f && (!kBoth || r != 0.f)) acc[a][b] = fmaf(l, r, acc[a][b]);
            }
        }
    }
}

// The tile's hidden layers (h1t, h2t) and outputs; samples past n count as zero
// inputs.  h2 of this thread's 4 samples x 4 units stays in `h2`.  Returns
// whether this thread met an input or a unit of h1 that is infinite or NaN.
__device__ __forceinline__ bool forward_tile(TileShared& s, TileGrad* gr, const __half* x, uint32_t first,
                                             uint32_t n, float (&h2)[4][4]) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    bool odd = false;
    for (int i = threadIdx.x; i < kTile * F; i += kThreads) {
        const uint32_t at = first + i / F;
        const float v = at < n ? __half2float(x[(uint64_t)at * F + i % F]) : 0.f;
        s.xt[i % F][i / F] = v;
        if (gr) { gr->x[i / F][i % F] = v; odd |= !isfinite(v); }
    }
    __syncthreads();
    float h1[4][4];
    #pragma unroll
    for (int a = 0; a < 4; ++a) {
        #pragma unroll
        for (int b = 0; b < 4; ++b) h1[a][b] = s.b1[4 * tx + b];
    }
    product<F>(s.xt, s.w1t, ty, tx, h1);
    #pragma unroll
    for (int a = 0; a < 4; ++a) {
        #pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float v = h1[a][b] > 0.f ? h1[a][b] : 0.f;
            s.h1t[4 * tx + b][4 * ty + a] = v;
            if (gr) { gr->h1[4 * ty + a][4 * tx + b] = v; odd |= !isfinite(v); }
        }
    }
    __syncthreads();
    #pragma unroll
    for (int a = 0; a < 4; ++a) {
        #pragma unroll
        for (int b = 0; b < 4; ++b) h2[a][b] = s.b2[4 * tx + b];
    }
    product<H>(s.h1t, s.w2t, ty, tx, h2);
    #pragma unroll
    for (int a = 0; a < 4; ++a) {
        #pragma unroll
        for (int b = 0; b < 4; ++b) {
            h2[a][b] = h2[a][b] > 0.f ? h2[a][b] : 0.f;
            s.h2t[4 * tx + b][4 * ty + a] = h2[a][b];
        }
    }
    __syncthreads();
    if (threadIdx.x < kTile) {
        float o = s.b3;
        #pragma unroll 8
        for (int j = 0; j < H; ++j) o = fmaf(s.w3[j], s.h2t[j][threadIdx.x], o);
        s.out[threadIdx.x] = o;
    }
    __syncthreads();
    return odd;
}

// Forward pass.  What bounds it: latency (a few thousand samples are a few
// tiles); one thread per sample ran its 5 000 multiply-adds one after the other.
__global__ void __launch_bounds__(kThreads) forward_kernel(const __half* w, const __half* x, uint32_t n,
                                                           float* out) {
    extern __shared__ __align__(16) unsigned char smem[];
    TileShared& s = *reinterpret_cast<TileShared*>(smem);
    load_weights(w, s);
    const uint32_t tiles = (n + kTile - 1) / kTile;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t first = t * kTile;
        float h2[4][4];
        forward_tile(s, nullptr, x, first, n, h2);
        if (threadIdx.x < kTile && first + threadIdx.x < n) out[first + threadIdx.x] = s.out[threadIdx.x];
        __syncthreads();
    }
}

// Forward and backward pass of the mean squared error over a block's tiles: the
// block's sums of the weight gradients and of e^2, in FP32 registers until the
// end, then NP + 1 values to part[block] (summed in a fixed order by
// gradient_sum_kernel; the last one is the loss).
//
// What bounds it: FP32 multiply-adds (33 738 samples: 1.05 GFLOP, 15 us at the
// chip's rate).  One thread per sample with one shared-memory atomic per sample
// and weight took 2.1 ms of device time; this takes 0.04.
__global__ void __launch_bounds__(kThreads) gradient_kernel(const __half* w, const __half* x, const float* y,
                                                            uint32_t n, float* part) {
    extern __shared__ __align__(16) unsigned char smem[];
    TileShared& s = *reinterpret_cast<TileShared*>(smem);
    TileGrad& g = *reinterpret_cast<TileGrad*>(smem + (sizeof(TileShared) + 15) / 16 * 16);
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    load_weights(w, s);
    bool odd_w = false;
    for (int i = tid; i < H * H; i += kThreads) {
        const float v = __half2float(w[OFF_W2 + i]);
        g.w2[i / H][i % H] = v;
        odd_w |= !isfinite(v);
    }
    float dw2[4][4] = {}, dw1[4] = {}, dw3[4] = {}, db2[4] = {};   // dw2: [4 ty + a][4 tx + b] = [j][q]
    float db1 = 0.f, db3 = 0.f, loss = 0.f;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t first = t * kTile;
        float h2[4][4];
        bool odd = forward_tile(s, &g, x, first, n, h2) || odd_w;
        if (tid < kTile) {
            const float e = first + tid < n ? s.out[tid] - y[first + tid] : 0.f;
            const float d = 2.f * e / (float)n;
            g.dout[tid] = d;
            loss += e * e / (float)n;
            db3 += d;
        }
        __syncthreads();
        // dh2 of this thread's 4 samples x 4 units
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float d = g.dout[4 * ty + a];
            const bool live = first + 4 * ty + a < n;     // (a sample past n adds nothing)
            #pragma unroll
            for (int b = 0; b < 4; ++b) {
                const float h = live ? h2[a][b] : 0.f;
                dw3[b] = fmaf(d, h, dw3[b]);
                const float v = h > 0.f ? d * s.w3[4 * tx + b] : 0.f;
                odd |= !isfinite(v);
                db2[b] += v;
                g.dh2[4 * ty + a][4 * tx + b] = v;
                s.h2t[4 * tx + b][4 * ty + a] = v;
            }
        }
        // a zero times an infinity is NaN, but a unit that is off, or an output that
        // is right, has no part in the gradient: such a tile (an input past FP16's
        // range, say) takes its products term by term
        odd = __syncthreads_or(odd);
        float dh1[4][4] = {};
        if (odd) {
            product_of_nonzeros<kTile, true>(g.dh2, g.h1, ty, tx, dw2);
            product_of_nonzeros<H, false>(s.h2t, g.w2, ty, tx, dh1);
        } else {
            product<kTile>(g.dh2, g.h1, ty, tx, dw2);
            product<H>(s.h2t, g.w2, ty, tx, dh1);
        }
        __syncthreads();   // every thread has read h1
        #pragma unroll
        for (int a = 0; a < 4; ++a) {
            #pragma unroll
            for (int b = 0; b < 4; ++b)
                g.h1[4 * ty + a][4 * tx + b] = s.h1t[4 * tx + b][4 * ty + a] > 0.f ? dh1[a][b] : 0.f;
        }
        __syncthreads();
        // dw1[q][f .. f + 3]: q = tid / 4, f = 4 (tid % 4)
        #pragma unroll 8
        for (int i = 0; i < kTile; ++i) {
            const float d = g.h1[i][tid >> 2];
            const float4 v = *reinterpret_cast<const float4*>(&g.x[i][4 * (tid & 3)]);
            if (odd && d == 0.f) continue;
            dw1[0] = fmaf(d, v.x, dw1[0]); dw1[1] = fmaf(d, v.y, dw1[1]);
            dw1[2] = fmaf(d, v.z, dw1[2]); dw1[3] = fmaf(d, v.w, dw1[3]);
            if ((tid & 3) == 0) db1 += d;
        }
        __syncthreads();   // before the next tile's loads
    }
    float* p = part + (uint64_t)blockIdx.x * (NP + 1);
    #pragma unroll
    for (int a = 0; a < 4; ++a) {
        #pragma unroll
        for (int b = 0; b < 4; ++b) p[OFF_W2 + (4 * ty + a) * H + 4 * tx + b] = dw2[a][b];
        p[OFF_W1 + (tid >> 2) * F + 4 * (tid & 3) + a] = dw1[a];
    }
    if ((tid & 3) == 0) p[OFF_B1 + (tid >> 2)] = db1;
    // sums over the 16 sample groups (ty), and over the samples
    #pragma unroll 1
    for (int b = 0; b < 4; ++b) {
        #pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            __syncthreads();
            g.red[tx * 16 + ty] = k ? db2[b] : dw3[b];
            __syncthreads();
            if (ty == 0) {
                float v = 0.f;
                for (int i = 0; i < 16; ++i) v += g.red[tx * 16 + i];
                p[(k ? OFF_B2 : OFF_W3) + 4 * tx + b] = v;
            }
        }
    }
    #pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        __syncthreads();
        g.red[tid] = k ? loss : db3;
        __syncthreads();
        if (tid == 0) {
            float v = 0.f;
            for (int i = 0; i < kTile; ++i) v += g.red[i];
            p[k ? NP : OFF_B3] = v;
        }
    }
}

// grad[p] = sum over blocks of part[.][p]; loss = the last column.  One warp per
// 8 parameters, 4 lanes each, so that the loads of a column overlap.
__global__ void gradient_sum_kernel(const float* part, uint32_t blocks, float* grad, float* loss) {
    const uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, lane = threadIdx.x & 3u;
    float v = 0.f;
    if (p <= NP) {
        #pragma unroll 4
        for (uint32_t i = lane; i < blocks; i += 4) v += part[(uint64_t)i * (NP + 1) + p];
    }
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    if (lane == 0 && p <= NP) *(p < NP ? grad + p : loss) = v;
}

// Adam step on the FP32 master weights; refreshes the FP16 copy.
__global__ void adam_kernel(float* master, __half* w, const float* grad, float* m, float* v,
                            float lr, float b1, float b2, float eps, float c1, float c2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NP) return;
    const float g = grad[p];
    const float mm = b1 * m[p] + (1.f - b1) * g;
    const float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    const float upd = lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    master[p] -= upd;
    w[p] = __float2half_rn(master[p]);
}

__global__ void to_half_kernel(const float* master, __half* w) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < NP) w[p] = __float2half_rn(master[p]);
}

__global__ void float_to_half_kernel(const float* in, __half* out, uint64_t n) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2half_rn(in[i]);
}

}  // namespace mlp
}  // namespace gmk
