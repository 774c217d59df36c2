// Data gradient of the descriptor's first convolution (conv1_1: 3 -> 64 channels, 3x3) on the
// 5th-generation tensor cores, through the normalisation and the 2x2 box downsample back to the
// renders (autograd of the reference's VGGLoss input, src/descriptor.py:7-79).
//
// As a 3x3 convolution 64 -> 3 channels it is 9 taps of an N = 16 product with 13 empty columns, and an
// MMA whose A operand starts inside a swizzle atom issues every 75 cycles whatever its N. Here the
// 9 taps x 3 channels are the columns of one N = 32 product instead: Y[q][tap, c] = sum_k g[q][k]
// w[tap][c][k] over a row of pixels q, 4 aligned MMAs per 128 pixels in place of 36, and the
// epilogue adds the 9 shifted results, out[p][c] = sum_tap Y[p + offset(tap)][tap, c]:
//   * along x by shuffles between the lanes that hold neighbouring pixels (a warp's edge pixels
//     pass through shared memory),
//   * along y in registers, each thread keeping its pixel column's sums of the two rows to come.
// What remains is reading g (128 bytes a pixel) once: 9 gradients of 256^2 take 25 us, the
// N = 16 convolution took 54.
//
// A block takes a strip of rows of one image and NX x 128 pixels of x (all of a map up to 256
// wide; wider maps in windows that overlap by two pixels): warp 0 loads the rows by TMA (128-byte
// swizzled pixel rows; the zero fill outside the image is the convolution's padding), one thread
// issues the MMAs into two TMEM buffers, 4 NX warps drain them. Small enough that two blocks share an
// SM. All waits are bounded: on timeout the kernel writes an error code to `err`, finishes
// without further waits and releases its TMEM.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <atomic>

#include "tc_ptx.cuh"

namespace svb {
namespace conv1g {

using namespace svb::tc;

constexpr int kStages = 3;
constexpr int kTileBytes = 128 * 128;  // 128 pixels x 64 channels BF16
constexpr int kCols = 32;              // 27 (tap, channel) columns, 5 empty
constexpr int kWBytes = kCols * 128;
enum GradError : int { kErrTma = 41, kErrMma = 42, kErrEpi = 43 };

template <int NX, bool DOWN>
__global__ void __launch_bounds__(64 + 128 * NX, 2)
conv1_grad_kernel(const __grid_constant__ CUtensorMap tmap_g, const __nv_bfloat16* __restrict__ w16,
                  const float* __restrict__ scale, float* __restrict__ dr, int H, int W, int rows, int windows,
                  int* err) {
  constexpr int NW = 4 * NX;  // epilogue warps, in pixel order
  constexpr uint32_t BUF = NX * kCols, TMEM_COLS = 2 * BUF;
  extern __shared__ uint8_t dsmem[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], tfull_bar[2], tempty_bar[2], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ float s_left[2][NW + 1][9], s_right[2][NW + 1][9];  // per row parity: what warp w's edge lanes take

  const uint32_t wbase = (smem_u32(dsmem) + 1023u) & ~1023u;
  const uint32_t abase = wbase + (uint32_t)kWBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int img = blockIdx.z;
  const int xw = windows == 1 ? 0 : (int)blockIdx.y * (128 * NX - 2) - 1;  // the window's first pixel
  const int ys = blockIdx.x * rows, ye = min(H, ys + rows);
  const int n_rows = ye - ys + 2;  // input rows ys - 1 .. ye

  // the weights as 32 K-major rows of 128 bytes, 128-byte swizzled: row 3 tap + c is w16[c][tap]
  for (int i = threadIdx.x; i < kCols * 8; i += blockDim.x) {
    const int n = i >> 3, j = i & 7;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n < 27) v = __ldg(reinterpret_cast<const uint4*>(w16 + ((n % 3) * 9 + n / 3) * 64) + j);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(wbase + (uint32_t)(n * 128 + ((j ^ (n & 7)) * 16))),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
  }
  fence_async_smem();  // read by the MMAs (async proxy); the barrier below orders them
  for (int i = threadIdx.x; i < 2 * (NW + 1) * 9; i += blockDim.x) {
    (&s_left[0][0][0])[i] = 0.0f;
    (&s_right[0][0][0])[i] = 0.0f;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tfull_bar[a]), 1);
      mbar_init(smem_u32(&tempty_bar[a]), NW);
    }
    mbar_init(smem_u32(&done_bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int j = 0; j < n_rows; ++j) {
        const int s = j % kStages;
        if (j >= kStages && !mbar_wait(smem_u32(&empty_bar[s]), ((uint32_t)(j / kStages) & 1u) ^ 1u, err, kErrTma)) break;
        const uint32_t fb = smem_u32(&full_bar[s]);
        mbar_expect_tx(fb, (uint32_t)(NX * kTileBytes));
#pragma unroll
        for (int m = 0; m < NX; ++m)
          tma_4d(abase + (uint32_t)((s * NX + m) * kTileBytes), &tmap_g, 0, xw + 128 * m, ys - 1 + j, img, fb);
        ++issued;
      }
      drain_loads(full_bar, issued, kStages);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16(128, kCols);
      for (int j = 0; j < n_rows; ++j) {
        const int s = j % kStages, a = j & 1;
        if (j >= 2 && !mbar_wait(smem_u32(&tempty_bar[a]), ((uint32_t)(j >> 1) & 1u) ^ 1u, err, kErrMma)) break;
        if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(j / kStages) & 1u, err, kErrMma)) break;
        fence_after();
#pragma unroll
        for (int m = 0; m < NX; ++m)
#pragma unroll
          for (int k = 0; k < 4; ++k)  // 16 channels (32 bytes) per MMA
            mma_bf16(tmem + (uint32_t)a * BUF + (uint32_t)(m * kCols),
                     sw128_desc(abase + (uint32_t)((s * NX + m) * kTileBytes) + 32u * k), sw128_desc(wbase + 32u * k),
                     idesc, k > 0 ? 1u : 0u);
        mma_commit(smem_u32(&empty_bar[s]));
        mma_commit(smem_u32(&tfull_bar[a]));
      }
      mma_commit(smem_u32(&done_bar));  // also on abort, so TMEM is idle before it is freed
    }
  } else {
    const int qw = warp & 3;            // the TMEM lane quadrant this warp may read
    const int m = (warp - 2) >> 2;      // its M-tile
    const int wi = 4 * m + qw;          // its place in pixel order
    const int px = 32 * wi + lane, x = xw + px;
    const bool inside = x >= 0 && x < W && (windows == 1 || (px >= 1 && px <= 128 * NX - 2));
    const float sc[3] = {__ldg(scale), __ldg(scale + 1), __ldg(scale + 2)};
    float p0[3] = {0.f, 0.f, 0.f}, p1[3] = {0.f, 0.f, 0.f};  // rows y - 1 and y so far, y = ys - 1 + j
    bool ok = true;
    for (int j = 0; j < n_rows; ++j) {
      const int a = j & 1;
      // every warp runs every row (the barrier below), with zeros once a wait has given up
      ok = ok && __all_sync(0xffffffffu, mbar_wait(smem_u32(&tfull_bar[a]), (uint32_t)(j >> 1) & 1u, err, kErrEpi)) &&
           *(volatile int*)err == 0;
      ok = __all_sync(0xffffffffu, ok);
      fence_after();
      uint32_t r[32];
      if (ok) {
        tmem_ld32(tmem + ((uint32_t)(qw * 32) << 16) + (uint32_t)a * BUF + (uint32_t)(m * kCols), r);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0u;
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[a]));
      // column (ky, kx, c) = 9 ky + 3 kx + c: kx = 0 goes to the pixel on the right, kx = 2 to the left
      if (lane == 31) {
#pragma unroll
        for (int i = 0; i < 9; ++i) s_left[a][wi + 1][i] = __uint_as_float(r[9 * (i / 3) + i % 3]);
      }
      if (lane == 0 && wi > 0) {
#pragma unroll
        for (int i = 0; i < 9; ++i) s_right[a][wi - 1][i] = __uint_as_float(r[9 * (i / 3) + 6 + i % 3]);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
      float h[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        float l = __shfl_up_sync(0xffffffffu, __uint_as_float(r[9 * (i / 3) + i % 3]), 1);
        float q = __shfl_down_sync(0xffffffffu, __uint_as_float(r[9 * (i / 3) + 6 + i % 3]), 1);
        if (lane == 0) l = s_left[a][wi][i];
        if (lane == 31) q = s_right[a][wi][i];
        h[i] = (l + __uint_as_float(r[9 * (i / 3) + 3 + i % 3])) + q;
      }
      // input row y = ys - 1 + j adds its ky = 2 part to output row y - 1, ky = 1 to y, ky = 0 to y + 1
      const int yo = ys + j - 2;
      if (j >= 2 && inside && ok) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float val = (p0[c] + h[6 + c]) * sc[c];
          if (DOWN) {
            float* o = dr + (((size_t)img * 3 + c) * 2 * H + 2 * yo) * (size_t)(2 * W) + 2 * x;
            *reinterpret_cast<float2*>(o) = make_float2(val, val);
            *reinterpret_cast<float2*>(o + 2 * W) = make_float2(val, val);
          } else {
            dr[(((size_t)img * 3 + c) * H + yo) * (size_t)W + x] = val;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        p0[c] = p1[c] + h[3 + c];
        p1[c] = h[c];
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    uint32_t it = 0;
    while (!mbar_try(smem_u32(&done_bar), 0u) && ++it < kSpin) {
    }
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

template <int NX, bool DOWN>
static int launch(const CUtensorMap& mg, const __nv_bfloat16* w16, const float* scale, float* dr, int n, int h, int w,
                  int* err, cudaStream_t st) {
  constexpr size_t smem = (size_t)kStages * NX * kTileBytes + kWBytes + 1024;
  auto kern = conv1_grad_kernel<NX, DOWN>;
  static std::atomic<bool> attr[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(SVBRDF_ERR_CUDA, "no usable device");
  if (!attr[dev].load()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return fail(SVBRDF_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(cudaGetLastError()));
    attr[dev].store(true);
  }
  const int sms = device_sm_count();
  const int windows = w <= 128 * NX ? 1 : (w + 128 * NX - 3) / (128 * NX - 2);
  // strips that make about two blocks per SM; each reads two rows more than it writes, so they have 4
  // rows or more (a column's last one what is left)
  const long long total = (long long)n * windows * h, slots = 2LL * (sms > 0 ? sms : 1);
  long long rows = (total + slots - 1) / slots;
  rows = rows < 4 ? 4 : rows > h ? h : rows;
  const dim3 grid((unsigned)((h + rows - 1) / rows), (unsigned)windows, (unsigned)n);
  kern<<<grid, 64 + 128 * NX, smem, st>>>(mg, w16, scale, dr, h, w, (int)rows, windows, err);
  return check_launch("conv1_grad_kernel");
}

}  // namespace conv1g
}  // namespace svb

using namespace svb;

extern "C" int svbrdf_desc_conv1_bwd_tc(const void* gz, const void* w16, const float* scale, float* dr, int n, int h,
                                        int w, int down, int* err, void* stream) {
  using namespace svb::conv1g;
  if (!gz || !w16 || !scale || !dr || !err) return fail(SVBRDF_ERR_INVALID, "conv1_bwd_tc: null argument");
  if (n < 1 || n > 65535 || h < 8 || w < 16 || h % 8 || w % 16)
    return fail(SVBRDF_ERR_UNSUPPORTED, "conv1_bwd_tc: H must be a multiple of 8 and W of 16 (got %dx%d)", h, w);
  if (((uintptr_t)gz | (uintptr_t)w16) % 16 || (uintptr_t)dr % 8)
    return fail(SVBRDF_ERR_INVALID, "conv1_bwd_tc: gz / w16 must be 16-byte aligned, dr 8-byte aligned");
  if ((long long)n * h * w * 64 >= (1LL << 40)) return fail(SVBRDF_ERR_UNSUPPORTED, "conv1_bwd_tc: tensor too large");
  PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  const int rc = svb::tc::get_tensor_map_encoder(&encode);
  if (rc) return rc;
  CUtensorMap mg;
  const cuuint64_t dims[4] = {64, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
  const cuuint64_t strides[3] = {64 * 2, (cuuint64_t)w * 64 * 2, (cuuint64_t)h * w * 64 * 2};
  const cuuint32_t box[4] = {64u, 128u, 1u, 1u};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const CUresult r = encode(&mg, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(gz), dims, strides, box, es,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(SVBRDF_ERR_CUDA, "cuTensorMapEncodeTiled(gz) failed: %d", (int)r);
  const __nv_bfloat16* wt = (const __nv_bfloat16*)w16;
  cudaStream_t st = (cudaStream_t)stream;
  if (w <= 128)
    return down ? launch<1, true>(mg, wt, scale, dr, n, h, w, err, st) : launch<1, false>(mg, wt, scale, dr, n, h, w, err, st);
  return down ? launch<2, true>(mg, wt, scale, dr, n, h, w, err, st) : launch<2, false>(mg, wt, scale, dr, n, h, w, err, st);
}
