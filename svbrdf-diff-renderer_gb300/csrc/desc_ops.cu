// Fused operations of the descriptor loss around the tensor-core convolutions (conv_tc.cu).
//
// The descriptor (src/descriptor.py:7-79) normalises the renders with ImageNet statistics
// (mean 0.485/0.456/0.406, std 0.229/0.224/0.255, :65-75), runs VGG19 features and compares
// hooked ReLU outputs. Here the renders are first 2x2 box-downsampled, and the stack up to
// conv4_1 runs in NHWC BF16. These kernels replace the elementwise glue:
//
//   desc_conv1_fwd_kernel  2x2 box downsample + normalise + conv1_1 (3 -> 64) + bias + ReLU,
//                          FP32 and BF16 NHWC outputs (the FP32 copy feeds the relu1_1 hook)
//   desc_pool_fwd_kernel   2x2 max-pool (or average pool), NHWC BF16
//   desc_pool_bwd_kernel   its backward (max: the first maximum of each window takes the
//                          gradient, as ATen's pool; average: a quarter to each) + optional
//                          hook gradient (given, or made from the hook's feature term) + ReLU mask
//   desc_feat_loss_kernel  sum of (f - t)^2 as per-block partials (a fixed-order sum), and
//                          optionally g = coef (f - t) + gram_grad, masked by f > 0
//   desc_loss_sums_kernel  weighted sums of loss partials (fixed order)
//   desc_conv1_bwd_kernel  conv1_1 data gradient, back through the normalisation and the
//                          downsample to d/d render
//
// Each is HBM-bound elementwise or small-stencil work: one read and one write per element.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "svbrdf_common.cuh"

namespace svb {
namespace desc {

__constant__ float c_mean[3] = {0.485f, 0.456f, 0.406f};
__constant__ float c_std[3] = {0.229f, 0.224f, 0.255f};  // the reference's blue std is 0.255

constexpr int kTile = 16;

// ---------------------------------------------------------------- conv1_1 forward
// A block computes kRep 8-row x 16-column pixel tiles one below the other, all 64 channels, with 256
// threads. Thread t owns channels 4 (t % 16) .. +3 of 8 pixels of a tile row (half (t / 16) % 2 of
// row t / 32), so the 16 threads of a half-warp store one pixel's 64 channels as one contiguous
// 256-byte run (128 bytes in BF16). The products run as packed FP32 pair FMAs (channels 4k, 4k+1
// and 4k+2, 4k+3), each lane rounded as a scalar FMA.
// Bound by the latency of its own loads when a block staged one tile (weights, then inputs, then
// arithmetic; 5 of a warp's 10 stalled cycles per instruction): the weights are staged once for the
// block's tiles and the next tile's inputs (and LOSS's first targets) are in flight during a
// tile's arithmetic. 9 renders of 512^2 (256^2 maps): 70 -> 60 us.
// LOSS: the feature term of this layer's hook as desc_feat_loss_kernel computes it, from the
// accumulators: d = f - t, partial[block] = sum d^2, g = coef d in BF16. The FP32 features are then
// not stored, and the term takes no pass of its own (63 + 65 us -> 80 us).
constexpr int kTileY = 8;
constexpr int kRep = 4;
constexpr int kConv1Threads = 256;
constexpr int kPx = 8;  // pixels per thread
template <bool DOWN, bool LOSS>
__global__ void __launch_bounds__(kConv1Threads, 3)
desc_conv1_fwd_kernel(const float* __restrict__ r, const float* __restrict__ w, const float* __restrict__ b,
                      float* __restrict__ out32, __nv_bfloat16* __restrict__ out16, int H, int W,
                      const float* __restrict__ target, float coef, __nv_bfloat16* __restrict__ g,
                      float* __restrict__ partial) {
  constexpr int kIn = 3 * (kTileY + 2) * (kTile + 2);  // inputs of a tile
  constexpr int kSlots = (kIn + kConv1Threads - 1) / kConv1Threads;
  constexpr int kRaw = DOWN ? 4 : 1;
  __shared__ float s_in[2][3][kTileY + 2][kTile + 2];
  __shared__ __align__(16) float s_w[27][64];  // [ci*9 + ky*3 + kx][co]
  __shared__ __align__(16) float s_b[64];
  __shared__ float s_red[kConv1Threads / 32];
  const int tid = threadIdx.x;
  const int v = blockIdx.z, x0 = blockIdx.x * kTile;
  const int RH = DOWN ? 2 * H : H, RW = DOWN ? 2 * W : W;
  float raw[kSlots][kRaw];
  // the raw renders under element i = tid + 256 u of the tile at y0 (its halo included)
  auto fetch = [&](int y0) {
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      const int i = tid + u * kConv1Threads;
      const int ci = i / ((kTileY + 2) * (kTile + 2)), rem = i % ((kTileY + 2) * (kTile + 2));
      const int gy = y0 + rem / (kTile + 2) - 1, gx = x0 + rem % (kTile + 2) - 1;
      if (i < kIn && gy >= 0 && gy < H && gx >= 0 && gx < W) {
        const float* rp = r + ((size_t)v * 3 + ci) * RH * RW;
        if constexpr (DOWN) {
          const float* q = rp + (size_t)(2 * gy) * RW + 2 * gx;
          raw[u][0] = __ldg(q); raw[u][1] = __ldg(q + 1); raw[u][2] = __ldg(q + RW); raw[u][3] = __ldg(q + RW + 1);
        } else {
          raw[u][0] = __ldg(rp + (size_t)gy * RW + gx);
        }
      }
    }
  };
  // ... normalised into buffer `to` (zero outside the image: the convolution's padding)
  auto stage = [&](int to, int y0) {
#pragma unroll
    for (int u = 0; u < kSlots; ++u) {
      const int i = tid + u * kConv1Threads;
      if (i >= kIn) continue;
      const int ci = i / ((kTileY + 2) * (kTile + 2)), rem = i % ((kTileY + 2) * (kTile + 2));
      const int ty = rem / (kTile + 2), tx = rem % (kTile + 2);
      const int gy = y0 + ty - 1, gx = x0 + tx - 1;
      float val = 0.0f;
      if (gy >= 0 && gy < H && gx >= 0 && gx < W) {
        float sv = raw[u][0];
        if constexpr (DOWN) sv = (raw[u][0] + raw[u][1] + raw[u][2] + raw[u][3]) * 0.25f;
        val = (sv - c_mean[ci]) / c_std[ci];
      }
      s_in[to][ci][ty][tx] = val;
    }
  };
  const int ybase = blockIdx.y * kRep * kTileY;
  fetch(ybase);
  for (int i = tid; i < 64 * 27; i += kConv1Threads) s_w[i >> 6][i & 63] = __ldg(w + (i & 63) * 27 + (i >> 6));
  if (tid < 64) s_b[tid] = b[tid];
  stage(0, ybase);
  __syncthreads();
  const int cg = tid & 15, row = tid >> 5, px0 = ((tid >> 4) & 1) * kPx;
  float sq = 0.0f;
  for (int rep = 0; rep < kRep; ++rep) {
    const int y0 = ybase + rep * kTileY;
    if (y0 >= H) break;
    const bool more = rep + 1 < kRep && y0 + kTileY < H;
    if (more) fetch(y0 + kTileY);
    const int y = y0 + row, x = x0 + px0;
    const size_t pix = ((size_t)v * H + y) * W + x;
    float sq_tile = 0.0f;  // a pixel's squares first, then a tile's: no sum of 128 terms in a row
    float4 tv[4];
    if (LOSS && y < H) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (x + u < W) tv[u] = __ldg(reinterpret_cast<const float4*>(target + (pix + u) * 64) + cg);
    }
    float2 acc[kPx][2];
    const float4 bias4 = reinterpret_cast<const float4*>(s_b)[cg];
#pragma unroll
    for (int px = 0; px < kPx; ++px) {
      acc[px][0] = make_float2(bias4.x, bias4.y);
      acc[px][1] = make_float2(bias4.z, bias4.w);
    }
#pragma unroll
    for (int ci = 0; ci < 3; ++ci)
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        // the inputs of this channel and kernel row, read once for the three kx taps
        float xr[kPx + 2];
#pragma unroll
        for (int i = 0; i < kPx + 2; ++i) xr[i] = s_in[rep & 1][ci][row + ky][px0 + i];
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          const float4 w4 = reinterpret_cast<const float4*>(s_w[ci * 9 + ky * 3 + kx])[cg];
          const float2 w01 = make_float2(w4.x, w4.y), w23 = make_float2(w4.z, w4.w);
#pragma unroll
          for (int px = 0; px < kPx; ++px) {
            const float2 x2 = make_float2(xr[px + kx], xr[px + kx]);
            acc[px][0] = __ffma2_rn(w01, x2, acc[px][0]);
            acc[px][1] = __ffma2_rn(w23, x2, acc[px][1]);
          }
        }
      }
    if (y < H) {
#pragma unroll
      for (int px = 0; px < kPx; ++px) {
        if (x + px >= W) break;
        const float a0 = fmaxf(acc[px][0].x, 0.f), a1 = fmaxf(acc[px][0].y, 0.f), a2 = fmaxf(acc[px][1].x, 0.f),
                    a3 = fmaxf(acc[px][1].y, 0.f);
        if (!LOSS) reinterpret_cast<float4*>(out32 + (pix + px) * 64)[cg] = make_float4(a0, a1, a2, a3);
        __nv_bfloat162 h0 = __floats2bfloat162_rn(a0, a1), h1 = __floats2bfloat162_rn(a2, a3);
        uint2 pk;
        pk.x = *reinterpret_cast<uint32_t*>(&h0);
        pk.y = *reinterpret_cast<uint32_t*>(&h1);
        reinterpret_cast<uint2*>(out16 + (pix + px) * 64)[cg] = pk;
        if (LOSS) {
          const float4 t4 = tv[px % 4];
          // the target four pixels on, in flight meanwhile
          if (px + 4 < kPx && x + px + 4 < W)
            tv[px % 4] = __ldg(reinterpret_cast<const float4*>(target + (pix + px + 4) * 64) + cg);
          const float d0 = a0 - t4.x, d1 = a1 - t4.y, d2 = a2 - t4.z, d3 = a3 - t4.w;
          sq_tile += fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, d3 * d3)));
          __nv_bfloat162 g0 = __floats2bfloat162_rn(coef * d0, coef * d1), g1 = __floats2bfloat162_rn(coef * d2, coef * d3);
          pk.x = *reinterpret_cast<uint32_t*>(&g0);
          pk.y = *reinterpret_cast<uint32_t*>(&g1);
          reinterpret_cast<uint2*>(g + (pix + px) * 64)[cg] = pk;
        }
      }
    }
    sq += sq_tile;
    // buffer (rep + 1) & 1 was last read in the previous tile, before that tile's barrier
    if (more) stage((rep + 1) & 1, y0 + kTileY);
    __syncthreads();
  }
  if (LOSS) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((tid & 31) == 0) s_red[tid >> 5] = sq;
    __syncthreads();
    if (tid == 0) {
      float t = 0.0f;
      for (int k = 0; k < kConv1Threads / 32; ++k) t += s_red[k];
      partial[((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// ---------------------------------------------------------------- conv1_1 backward
// d render = conv1_1's data gradient (3 x 3, 64 -> 3 channels), through the normalisation
// and the 2x2 box downsample. A block takes a 16 x 16 tile of the 256-pixel side; each of its
// 128 threads computes 2 adjacent pixels of one row, so every weight pair and every input
// column read from shared memory serves up to 2 pixels (per channel pair and kernel row: 4
// input values and 9 weight pairs for 36 FMAs).
template <bool DOWN>
__global__ void __launch_bounds__(128) desc_conv1_bwd_kernel(const __nv_bfloat16* __restrict__ gz,
                                                            const float* __restrict__ w, float* __restrict__ gr,
                                                            int H, int W) {
  __shared__ __nv_bfloat162 s_g[32][kTile + 2][kTile + 2];  // gz tile, channel pairs outermost
  __shared__ __align__(8) float s_w[27][64];                 // [ci*9 + ky*3 + kx][co]
  const int tid = threadIdx.x;
  const int v = blockIdx.z, y0 = blockIdx.y * kTile, x0 = blockIdx.x * kTile;
  for (int i = tid; i < 64 * 27; i += 128) s_w[i % 27][i / 27] = w[i];
  // rows y0-1 .. y0+16 and columns x0-1 .. x0+16 of gz, 8 channels per step
  for (int i = tid; i < (kTile + 2) * (kTile + 2) * 8; i += 128) {
    const int p = i / 8, c8 = i % 8;
    const int ty = p / (kTile + 2), tx = p % (kTile + 2);
    const int gy = y0 + ty - 1, gx = x0 + tx - 1;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (gy >= 0 && gy < H && gx >= 0 && gx < W)
      val = *reinterpret_cast<const uint4*>(gz + (((size_t)v * H + gy) * W + gx) * 64 + c8 * 8);
    const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&val);
#pragma unroll
    for (int j = 0; j < 4; ++j) s_g[c8 * 4 + j][ty][tx] = e[j];
  }
  __syncthreads();
  const int ty = tid / 8, tx0 = 2 * (tid % 8);  // pixels (ty, tx0 .. tx0 + 1) of the tile
  float d[2][3];
#pragma unroll
  for (int q = 0; q < 2; ++q) d[q][0] = d[q][1] = d[q][2] = 0.f;
#pragma unroll 2
  for (int c2 = 0; c2 < 32; ++c2) {
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      // gz at output (y + 1 - ky, x + 1 - kx) = tile (ty + 2 - ky, tx + 2 - kx): columns tx0 .. tx0 + 3
      float2 g[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) g[j] = __bfloat1622float2(s_g[c2][ty + 2 - ky][tx0 + j]);
#pragma unroll
      for (int kx = 0; kx < 3; ++kx) {
#pragma unroll
        for (int ci = 0; ci < 3; ++ci) {
          const float2 wv = reinterpret_cast<const float2*>(s_w[ci * 9 + ky * 3 + kx])[c2];
#pragma unroll
          for (int q = 0; q < 2; ++q) d[q][ci] = fmaf(wv.y, g[q + 2 - kx].y, fmaf(wv.x, g[q + 2 - kx].x, d[q][ci]));
        }
      }
    }
  }
  const int y = y0 + ty, x = x0 + tx0;
  if (y >= H) return;
  const int RH = DOWN ? 2 * H : H, RW = DOWN ? 2 * W : W;
#pragma unroll
  for (int ci = 0; ci < 3; ++ci) {
    float* rp = gr + ((size_t)v * 3 + ci) * RH * RW;
    const float is = 1.0f / c_std[ci];
    float gq[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) gq[q] = d[q][ci] * is;
    if (DOWN) {
      if (x + 1 < W && RW % 4 == 0 && ((uintptr_t)rp & 15u) == 0) {  // 16-byte aligned rows
        const float4 a = make_float4(0.25f * gq[0], 0.25f * gq[0], 0.25f * gq[1], 0.25f * gq[1]);
        *reinterpret_cast<float4*>(rp + (size_t)(2 * y) * RW + 2 * x) = a;
        *reinterpret_cast<float4*>(rp + (size_t)(2 * y + 1) * RW + 2 * x) = a;
      } else {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (x + q >= W) break;
          const float qv = 0.25f * gq[q];
          *reinterpret_cast<float2*>(rp + (size_t)(2 * y) * RW + 2 * (x + q)) = make_float2(qv, qv);
          *reinterpret_cast<float2*>(rp + (size_t)(2 * y + 1) * RW + 2 * (x + q)) = make_float2(qv, qv);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (x + q < W) rp[(size_t)y * RW + x + q] = gq[q];
    }
  }
}

// ---------------------------------------------------------------- 2x2 max-pool
__device__ __forceinline__ void bf8_load(const __nv_bfloat16* p, float f[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(h[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
__device__ __forceinline__ void bf8_store(__nv_bfloat16* p, const float f[8]) {
  uint4 u;
  uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
    w[j] = *reinterpret_cast<uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = u;
}

// x [V, H, W, C] -> y [V, H/2, W/2, C]; one thread per output pixel and 8 channels.
// AVG: the window's mean (the reference's VGGLoss swaps VGG19's max-pools for 2x2 average
// pools, src/descriptor.py:16-19), summed in row-major order in FP32 then halved twice.
template <bool AVG>
__global__ void desc_pool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int V, int H,
                                     int W, int C) {
  // grid (ceil(Wo C8 / 256), V Ho): block row (v, yo); thread q of the row is (xo, c8)
  const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
  const int v = blockIdx.y / Ho, yo = blockIdx.y % Ho;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < Wo * C8; q += gridDim.x * blockDim.x) {
    const int c8 = q % C8, xo = q / C8;
    const size_t p = ((size_t)v * Ho + yo) * Wo + xo;
    const __nv_bfloat16* base = x + (((size_t)v * H + 2 * yo) * W + 2 * xo) * C + c8 * 8;
    float m[8], t[8];
    bf8_load(base, m);
    const size_t offs[3] = {(size_t)C, (size_t)W * C, (size_t)W * C + C};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      bf8_load(base + offs[k], t);
#pragma unroll
      for (int j = 0; j < 8; ++j) m[j] = AVG ? m[j] + t[j] : (t[j] > m[j] ? t[j] : m[j]);
    }
    if (AVG) {
#pragma unroll
      for (int j = 0; j < 8; ++j) m[j] *= 0.25f;
    }
    bf8_store(y + p * C + c8 * 8, m);
  }
}

// gx = (pool-route(gy) + addend) * (x > 0). x is the pool's input, a ReLU output, so x > 0 is
// that ReLU's mask. Max-pool: the window's first maximum in row-major order takes the
// gradient. AVG: every element of the window takes gy / 4. Each thread issues all of its loads
// (the window's x, gy, the window's addend: nine 16-byte loads) before any arithmetic, keeping
// them as raw BF16 until use.
// LOSS: the addend is not read but made here, where the hook's feature x is read anyway, as
// desc_feat_loss_kernel computes it: d = x - t with t the BF16 target that `addend` points to, coef d
// rounded to BF16, partial[block] = sum d^2. The hook's term then takes no pass of its own (9 maps of
// 256^2 x 64, relu1_2: 43 + 37 -> 43 us, HBM-bound as both were).
__device__ __forceinline__ float2 bf2f(const uint4& u, int e) {
  return __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&u)[e]);
}
template <bool AVG, bool LOSS>
__global__ void __launch_bounds__(256) desc_pool_bwd_kernel(const __nv_bfloat16* __restrict__ gy,
                                                            const __nv_bfloat16* __restrict__ x,
                                                            const __nv_bfloat16* __restrict__ addend,
                                                            __nv_bfloat16* __restrict__ gx, int V, int H, int W,
                                                            int C, float coef, float* __restrict__ partial) {
  // grid (ceil(Wo C8 / 256), V Ho): block row (v, yo); thread t of the row is (xo, c8)
  const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
  const int v = blockIdx.y / Ho, yo = blockIdx.y % Ho;
  float sq = 0.0f;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < Wo * C8; t += gridDim.x * blockDim.x) {
    const int c8 = t % C8, xo = t / C8;
    const size_t p = ((size_t)v * Ho + yo) * Wo + xo;
    const size_t b0 = (((size_t)v * H + 2 * yo) * W + 2 * xo) * C + c8 * 8;
    const size_t offs[4] = {0, (size_t)C, (size_t)W * C, (size_t)W * C + C};
    uint4 xr[4], ar[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) xr[k] = __ldg(reinterpret_cast<const uint4*>(x + b0 + offs[k]));
    const uint4 gr = __ldg(reinterpret_cast<const uint4*>(gy + p * C + c8 * 8));
    if (LOSS || addend) {
#pragma unroll
      for (int k = 0; k < 4; ++k) ar[k] = __ldg(reinterpret_cast<const uint4*>(addend + b0 + offs[k]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) ar[k] = make_uint4(0u, 0u, 0u, 0u);  // BF16 zeros
    }
    uint4 o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {  // channel pairs 2e, 2e + 1
      const float2 g = bf2f(gr, e);
      float2 xv[4];
      float sq_pair = 0.0f;  // the pair's eight squares first
#pragma unroll
      for (int k = 0; k < 4; ++k) xv[k] = bf2f(xr[k], e);
      int amx = 0, amy = 0;
      if (!AVG) {
        float mx = xv[0].x, my = xv[0].y;
#pragma unroll
        for (int k = 1; k < 4; ++k) {
          if (xv[k].x > mx) { mx = xv[k].x; amx = k; }
          if (xv[k].y > my) { my = xv[k].y; amy = k; }
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 ad = bf2f(ar[k], e);
        if constexpr (LOSS) {
          const float2 d = make_float2(xv[k].x - ad.x, xv[k].y - ad.y);
          sq_pair = fmaf(d.x, d.x, sq_pair);
          sq_pair = fmaf(d.y, d.y, sq_pair);
          ad = __bfloat1622float2(__floats2bfloat162_rn(coef * d.x, coef * d.y));
        }
        float vx = AVG ? 0.25f * g.x : (amx == k ? g.x : 0.0f);
        float vy = AVG ? 0.25f * g.y : (amy == k ? g.y : 0.0f);
        vx += ad.x;
        vy += ad.y;
        const __nv_bfloat162 h = __floats2bfloat162_rn(xv[k].x > 0.0f ? vx : 0.0f, xv[k].y > 0.0f ? vy : 0.0f);
        reinterpret_cast<uint32_t*>(&o[k])[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      if constexpr (LOSS) sq += sq_pair;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(gx + b0 + offs[k]) = o[k];
  }
  if constexpr (LOSS) {
    __shared__ float s_red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      float s = 0.0f;
      for (int w = 0; w < 8; ++w) s += s_red[w];
      partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
    }
  }
}

// ---------------------------------------------------------------- feature loss
constexpr int kLossThreads = 256;
constexpr int kLossBlocks = 608;  // one wave of 4 per SM

__device__ __forceinline__ float ld(const float* p, long long i) { return __ldg(p + i); }
__device__ __forceinline__ float ld(const __nv_bfloat16* p, long long i) { return __bfloat162float(p[i]); }
// Eight elements from a 16-byte aligned address.
__device__ __forceinline__ void ld8(const float* p, float v[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float v[8]) { bf8_load(p, v); }

// partial[b] = sum over block b's elements of (f - t)^2; if g: g = coef (f - t) + gram_grad, times
// (f > 0) when `mask`. WIDE (n a multiple of 8, 16-byte aligned maps): a thread takes eight
// elements, two such steps in flight; HBM-bound, where one element at a time (2- and 4-byte
// accesses) took 78 us for the three BF16 hooks of the reference stack on 9 renders of 256^2, 62 so.
// Otherwise elements b T + t, step B T.
template <typename TF, typename TT, bool WIDE>
__global__ void __launch_bounds__(kLossThreads, 4)
desc_feat_loss_kernel(const TF* __restrict__ f, const TT* __restrict__ t, const float* __restrict__ gram_grad,
                      float coef, int mask, __nv_bfloat16* __restrict__ g, float* __restrict__ partial, long long n) {
  __shared__ float s_red[kLossThreads / 32];
  constexpr int E = WIDE ? 8 : 1, U = 2;
  float acc[U] = {};  // one per step in flight, and a step's eight squares first among themselves
  const long long step = (long long)kLossBlocks * kLossThreads * E;
  for (long long i0 = (blockIdx.x * (long long)kLossThreads + threadIdx.x) * E; i0 < n; i0 += U * step) {
    float fv[U][E], tv[U][E], gg[U][E];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * step;
#pragma unroll
      for (int e = 0; e < E; ++e) gg[u][e] = 0.0f;
      if (i >= n) continue;
      if constexpr (WIDE) {
        ld8(f + i, fv[u]);
        ld8(t + i, tv[u]);
        if (gram_grad) ld8(gram_grad + i, gg[u]);
      } else {
        fv[u][0] = ld(f, i);
        tv[u][0] = ld(t, i);
        if (gram_grad) gg[u][0] = ld(gram_grad, i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * step;
      if (i >= n) continue;
      float gv[E], sq = WIDE ? 0.0f : acc[u];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float d = fv[u][e] - tv[u][e];
        sq = fmaf(d, d, sq);
        gv[e] = gram_grad ? fmaf(coef, d, gg[u][e]) : coef * d;
        if (mask && !(fv[u][e] > 0.0f)) gv[e] = 0.0f;
      }
      acc[u] = WIDE ? acc[u] + sq : sq;
      if (!g) continue;
      if constexpr (WIDE) bf8_store(g + i, gv);
      else g[i] = __float2bfloat16_rn(gv[0]);
    }
  }
  if (partial) {
#pragma unroll
    for (int u = 1; u < U; ++u) acc[0] += acc[u];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = acc[0];
    __syncthreads();
    if (threadIdx.x == 0) {
      float s = 0.0f;
      for (int w = 0; w < kLossThreads / 32; ++w) s += s_red[w];
      partial[blockIdx.x] = s;
    }
  }
}

// ---------------------------------------------------------------- loss sums
// out[j] = sum over segments s of group j of w_s x (sum of the segment's floats), added in a
// fixed order by one block. The segments are cut into units of 256 floats; warp w takes units w,
// w + 32, ..., three at a time, eight loads a lane each, and a lane adds its terms of a segment in
// FP32 (a few dozen). The lanes' totals are added as FP32 pairs (sum, rounding error), so that the
// warp's share is as good as in double, and the shares are added and weighted in double, one warp
// per segment: a double-precision instruction holds this part's FP64 pipe for 16 cycles a warp, and
// with every thread keeping its totals in double those instructions were the kernel's 14 us
// (8 segments, 46,000 floats; about 10 us so).
constexpr int kMaxLossSegs = 16;
constexpr int kLossSumThreads = 1024;
struct LossSegs {
  long long off[kMaxLossSegs];
  long long len[kMaxLossSegs];
  double w[kMaxLossSegs];
  int group[kMaxLossSegs];
  int n;
};
__global__ void __launch_bounds__(kLossSumThreads) desc_loss_sums_kernel(const float* __restrict__ buf, LossSegs segs,
                                                                          float* __restrict__ out) {
  constexpr int kWarps = kLossSumThreads / 32, kU = 3;  // units of a warp in flight
  static_assert(kWarps == 32 && kMaxLossSegs <= kWarps, "one lane per warp's share, one warp per segment");
  __shared__ float2 share[kMaxLossSegs][kWarps];
  __shared__ unsigned in_double[kMaxLossSegs];  // bit w: warp w's share of the segment is a double's bits
  __shared__ double total[kMaxLossSegs];
  if (threadIdx.x < kMaxLossSegs) in_double[threadIdx.x] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long unit = warp;  // of this warp, counted from the start of segment k
  for (int k = 0; k < segs.n; ++k) {
    const long long len = segs.len[k], units = (len + 255) / 256;
    const float* p = buf + segs.off[k];
    float sk = 0.0f;
    for (; unit < units; unit += kU * kWarps) {
      float q[kU][8];
#pragma unroll
      for (int a = 0; a < kU; ++a)
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const long long i = (unit + a * kWarps) * 256 + lane + 32 * u;
          q[a][u] = i < len ? __ldg(p + i) : 0.0f;
        }
#pragma unroll
      for (int a = 0; a < kU; ++a)
        sk += ((q[a][0] + q[a][1]) + (q[a][2] + q[a][3])) + ((q[a][4] + q[a][5]) + (q[a][6] + q[a][7]));
    }
    while (unit >= units + kWarps) unit -= kWarps;  // the first of its units past the segment's end
    unit -= units;
    const float own = sk;
    float lo = 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float b = __shfl_xor_sync(0xffffffffu, sk, o), bl = __shfl_xor_sync(0xffffffffu, lo, o);
      const float s = sk + b, bb = s - sk;  // Knuth's two-sum: s + e = sk + b exactly
      lo += bl + ((sk - (s - bb)) + (b - bb));
      sk = s;
    }
    if (fabsf(sk) <= 3.402823466e+38f) {  // every lane holds the same sum
      if (lane == 0) share[k][warp] = make_float2(sk, lo);
    } else {
      // lane totals whose sum FP32 does not hold, or an infinity or NaN among them: in double
      double d = (double)own;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (lane == 0) {
        share[k][warp] = make_float2(__int_as_float(__double2loint(d)), __int_as_float(__double2hiint(d)));
        atomicOr(&in_double[k], 1u << warp);
      }
    }
  }
  __syncthreads();
  if (warp < segs.n) {
    const float2 sh = share[warp][lane];
    double t = (in_double[warp] >> lane) & 1u ? __hiloint2double(__float_as_int(sh.y), __float_as_int(sh.x))
                                              : (double)sh.x + (double)sh.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) total[warp] = segs.w[warp] * t;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int k = 0; k < segs.n; ++k)
      if (segs.group[k] == (int)threadIdx.x) t += total[k];
    out[threadIdx.x] = (float)t;
  }
}

}  // namespace desc
}  // namespace svb

using namespace svb;
using namespace svb::desc;

static dim3 conv1_grid(int v, int h, int w) {
  return dim3((w + kTile - 1) / kTile, (h + kTileY * kRep - 1) / (kTileY * kRep), v);
}

template <bool LOSS>
static int conv1_fwd(const float* renders, const float* weight, const float* bias, float* out_f32, void* out_bf16,
                     int v, int h, int w, int downsample, const float* target, float coef, void* g, float* partial,
                     void* stream) {
  if (v > 65535 || (h + kTileY - 1) / kTileY > 65535) return fail(SVBRDF_ERR_UNSUPPORTED, "conv1_fwd: too large");
  const dim3 grid = conv1_grid(v, h, w);
  cudaStream_t st = (cudaStream_t)stream;
  __nv_bfloat16 *o16 = (__nv_bfloat16*)out_bf16, *g16 = (__nv_bfloat16*)g;
  if (downsample)
    desc_conv1_fwd_kernel<true, LOSS><<<grid, kConv1Threads, 0, st>>>(renders, weight, bias, out_f32, o16, h, w, target, coef,
                                                            g16, partial);
  else
    desc_conv1_fwd_kernel<false, LOSS><<<grid, kConv1Threads, 0, st>>>(renders, weight, bias, out_f32, o16, h, w, target, coef,
                                                             g16, partial);
  return check_launch("desc_conv1_fwd_kernel");
}

static dim3 pool_grid(int v, int h, int w, int c) {
  return dim3((unsigned)(((w / 2) * (c / 8) + 255) / 256), (unsigned)(v * (h / 2)));
}

template <bool AVG>
static int pool_fwd(const void* x, void* y, int v, int h, int w, int c, void* stream) {
  if (!x || !y) return fail(SVBRDF_ERR_INVALID, "null pointer");
  if (v < 1 || h < 2 || w < 2 || h % 2 || w % 2 || c < 8 || c % 8)
    return fail(SVBRDF_ERR_UNSUPPORTED, "pool: even H, W and C a multiple of 8 needed");
  if (((uintptr_t)x | (uintptr_t)y) % 16) return fail(SVBRDF_ERR_INVALID, "pool: 16-byte alignment needed");
  if ((long long)v * (h / 2) > 65535 || (long long)(w / 2) * (c / 8) >= (1LL << 30))
    return fail(SVBRDF_ERR_UNSUPPORTED, "pool: too large");
  desc_pool_fwd_kernel<AVG><<<pool_grid(v, h, w, c), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, v, h, w, c);
  return check_launch("desc_pool_fwd_kernel");
}

template <bool AVG, bool LOSS>
static int pool_bwd(const void* gy, const void* x, const void* addend, void* gx, int v, int h, int w, int c,
                    float coef, float* partial, void* stream) {
  if (!gy || !x || !gx || (LOSS && (!addend || !partial))) return fail(SVBRDF_ERR_INVALID, "null pointer");
  if (v < 1 || h < 2 || w < 2 || h % 2 || w % 2 || c < 8 || c % 8)
    return fail(SVBRDF_ERR_UNSUPPORTED, "pool: even H, W and C a multiple of 8 needed");
  if (((uintptr_t)gy | (uintptr_t)x | (uintptr_t)addend | (uintptr_t)gx) % 16)
    return fail(SVBRDF_ERR_INVALID, "pool: 16-byte alignment needed");
  if ((long long)v * (h / 2) > 65535 || (long long)(w / 2) * (c / 8) >= (1LL << 30))
    return fail(SVBRDF_ERR_UNSUPPORTED, "pool: too large");
  desc_pool_bwd_kernel<AVG, LOSS><<<pool_grid(v, h, w, c), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)gy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)addend, (__nv_bfloat16*)gx, v, h, w,
      c, coef, partial);
  return check_launch("desc_pool_bwd_kernel");
}

extern "C" {

int svbrdf_desc_partials() { return kLossBlocks; }

int svbrdf_desc_conv1_fwd(const float* renders, const float* weight, const float* bias, float* out_f32,
                          void* out_bf16, int v, int h, int w, int downsample, void* stream) {
  if (!renders || !weight || !bias || !out_f32 || !out_bf16) return fail(SVBRDF_ERR_INVALID, "null pointer");
  if (v < 1 || h < 1 || w < 1) return fail(SVBRDF_ERR_INVALID, "bad shape");
  if (((uintptr_t)out_f32 | (uintptr_t)out_bf16) % 16) return fail(SVBRDF_ERR_INVALID, "outputs must be 16-byte aligned");
  return conv1_fwd<false>(renders, weight, bias, out_f32, out_bf16, v, h, w, downsample, nullptr, 0.0f, nullptr,
                          nullptr, stream);
}

long long svbrdf_desc_conv1_loss_partials(int v, int h, int w) {
  if (v < 1 || h < 1 || w < 1) return 0;
  const dim3 g = conv1_grid(v, h, w);
  return (long long)g.x * g.y * g.z;
}

int svbrdf_desc_conv1_loss(const float* renders, const float* weight, const float* bias, void* out_bf16, int v, int h,
                           int w, int downsample, const float* target, float coef, void* g, float* partial,
                           void* stream) {
  if (!renders || !weight || !bias || !out_bf16 || !target || !g || !partial)
    return fail(SVBRDF_ERR_INVALID, "conv1_loss: null pointer");
  if (v < 1 || h < 1 || w < 1) return fail(SVBRDF_ERR_INVALID, "bad shape");
  if (((uintptr_t)out_bf16 | (uintptr_t)target | (uintptr_t)g) % 16)
    return fail(SVBRDF_ERR_INVALID, "conv1_loss: 16-byte alignment");
  return conv1_fwd<true>(renders, weight, bias, nullptr, out_bf16, v, h, w, downsample, target, coef, g, partial,
                         stream);
}

int svbrdf_desc_conv1_bwd(const void* gz, const float* weight, float* grad_renders, int v, int h, int w, int downsample,
                          void* stream) {
  if (!gz || !weight || !grad_renders) return fail(SVBRDF_ERR_INVALID, "null pointer");
  if (v < 1 || h < 1 || w < 1) return fail(SVBRDF_ERR_INVALID, "bad shape");
  if ((uintptr_t)gz % 16 || (downsample && (uintptr_t)grad_renders % 8))
    return fail(SVBRDF_ERR_INVALID, "misaligned gz/grad_renders");
  dim3 grid((w + kTile - 1) / kTile, (h + kTile - 1) / kTile, v), block(128);
  cudaStream_t st = (cudaStream_t)stream;
  if (downsample)
    desc_conv1_bwd_kernel<true><<<grid, block, 0, st>>>((const __nv_bfloat16*)gz, weight, grad_renders, h, w);
  else
    desc_conv1_bwd_kernel<false><<<grid, block, 0, st>>>((const __nv_bfloat16*)gz, weight, grad_renders, h, w);
  return check_launch("desc_conv1_bwd_kernel");
}

int svbrdf_desc_pool_fwd(const void* x, void* y, int v, int h, int w, int c, void* stream) {
  return pool_fwd<false>(x, y, v, h, w, c, stream);
}

int svbrdf_desc_pool_bwd(const void* gy, const void* x, const void* addend, void* gx, int v, int h, int w, int c,
                         void* stream) {
  return pool_bwd<false, false>(gy, x, addend, gx, v, h, w, c, 0.0f, nullptr, stream);
}

int svbrdf_desc_avgpool_fwd(const void* x, void* y, int v, int h, int w, int c, void* stream) {
  return pool_fwd<true>(x, y, v, h, w, c, stream);
}

int svbrdf_desc_avgpool_bwd(const void* gy, const void* x, const void* addend, void* gx, int v, int h, int w, int c,
                            void* stream) {
  return pool_bwd<true, false>(gy, x, addend, gx, v, h, w, c, 0.0f, nullptr, stream);
}

long long svbrdf_desc_pool_bwd_loss_partials(int v, int h, int w, int c) {
  if (v < 1 || h < 2 || w < 2 || c < 8) return 0;
  const dim3 g = pool_grid(v, h, w, c);
  return (long long)g.x * g.y;
}

int svbrdf_desc_pool_bwd_loss(const void* gy, const void* x, const void* target, float coef, void* gx, float* partial,
                              int v, int h, int w, int c, int avg, void* stream) {
  return avg ? pool_bwd<true, true>(gy, x, target, gx, v, h, w, c, coef, partial, stream)
             : pool_bwd<false, true>(gy, x, target, gx, v, h, w, c, coef, partial, stream);
}

int svbrdf_desc_feat_loss(const void* f, int dtypes, const void* t, const float* gram_grad, float coef, int mask,
                          void* g, float* partial, long long n, void* stream) {
  if (!f || !t || n < 1) return fail(SVBRDF_ERR_INVALID, "null pointer or empty");
  if (dtypes < 0 || dtypes > 3) dtypes = 1;  // the flag that the argument was: any non-zero value, f BF16
  cudaStream_t st = (cudaStream_t)stream;
  const bool wide = n % 8 == 0 && (((uintptr_t)f | (uintptr_t)t | (uintptr_t)gram_grad | (uintptr_t)g) & 15) == 0;
#define SVB_FL(TF, TT, WIDE)                                                                        \
  desc_feat_loss_kernel<TF, TT, WIDE><<<kLossBlocks, kLossThreads, 0, st>>>(                        \
      (const TF*)f, (const TT*)t, gram_grad, coef, mask, (__nv_bfloat16*)g, partial, n)
#define SVB_FLW(TF, TT)            \
  if (wide) SVB_FL(TF, TT, true);  \
  else SVB_FL(TF, TT, false)
  switch (dtypes) {
    case 0: SVB_FLW(float, float); break;
    case 1: SVB_FLW(__nv_bfloat16, float); break;
    case 2: SVB_FLW(float, __nv_bfloat16); break;
    default: SVB_FLW(__nv_bfloat16, __nv_bfloat16); break;
  }
#undef SVB_FLW
#undef SVB_FL
  return check_launch("desc_feat_loss_kernel");
}

int svbrdf_desc_loss_sums(const float* buf, int n_segs, const long long* offsets, const long long* lengths,
                          const double* weights, const int* groups, float* out, void* stream) {
  if (!buf || !out || !offsets || !lengths || !weights || !groups) return fail(SVBRDF_ERR_INVALID, "null pointer");
  if (n_segs < 1 || n_segs > kMaxLossSegs)
    return fail(SVBRDF_ERR_UNSUPPORTED, "loss sums: 1 to %d segments (got %d)", kMaxLossSegs, n_segs);
  LossSegs segs;
  segs.n = n_segs;
  for (int k = 0; k < n_segs; ++k) {
    if (offsets[k] < 0 || lengths[k] < 0 || (groups[k] != 0 && groups[k] != 1))
      return fail(SVBRDF_ERR_INVALID, "loss sums: bad segment %d", k);
    segs.off[k] = offsets[k];
    segs.len[k] = lengths[k];
    segs.w[k] = weights[k];
    segs.group[k] = groups[k];
  }
  desc_loss_sums_kernel<<<1, kLossSumThreads, 0, (cudaStream_t)stream>>>(buf, segs, out);
  return check_launch("desc_loss_sums_kernel");
}

}  // extern "C"
