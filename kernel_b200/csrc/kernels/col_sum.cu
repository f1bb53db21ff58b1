// Column sums of a bf16 matrix in fp32 (bias gradients): out[c] = sum_r x[r, c].
//
// Bound by memory: x is read once, 16 bytes per thread, 512 contiguous bytes per warp.
// A CTA takes 256 columns and a contiguous range of rows; with several row ranges a
// second, small launch adds their fp32 partials in ascending order, so the result does
// not depend on timing.  8192 x 29568: 74 us (6.6 TB/s) with the second launch, against 804 us for a
// cast to fp32, a library reduction and a cast back; 8192 x 8192 23 and 244.
// One wave of the CTAs that fit: with eight CTAs asked for per SM, of which four fit, the last wave was mostly empty (116 and 28 us).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../include/kb200.h"

namespace {

constexpr int COLS = 256;   // columns of a CTA: 32 lanes x 8
constexpr int WARPS = 8;
constexpr int UNROLL = 8;   // rows in flight per warp
constexpr int CTAS = 4;     // resident per SM

__global__ void __launch_bounds__(32 * WARPS, CTAS) col_sum_kernel(const __nv_bfloat16* x, int rows, int cols, int rows_per,
                                                              float* partial, __nv_bfloat16* out) {
  __shared__ float s_sum[WARPS][COLS];
  kb::wait_for_previous_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * COLS + lane * 8;
  const int r1 = min(rows, static_cast<int>(blockIdx.y + 1) * rows_per);
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  if (c < cols) {
    for (int r = blockIdx.y * rows_per + warp; r < r1; r += UNROLL * WARPS) {
      uint4 v[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int row = r + u * WARPS;
        v[u] = row < r1 ? kb::ld_stream_v4(x + static_cast<size_t>(row) * cols + c) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = kb::unpack_bf16x2(w[e]);
          acc[2 * e] += f.x;
          acc[2 * e + 1] += f.y;
        }
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) s_sum[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  const int col = blockIdx.x * COLS + threadIdx.x;
  if (col < cols) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) sum += s_sum[w][threadIdx.x];
    if (partial != nullptr) partial[static_cast<size_t>(blockIdx.y) * cols + col] = sum;
    else out[col] = __float2bfloat16_rn(sum);
  }
}

__global__ void __launch_bounds__(256) col_sum_finish_kernel(const float* partial, int parts, int cols, __nv_bfloat16* out) {
  kb::wait_for_previous_launch();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= cols) return;
  float sum = 0.f;
  for (int i = 0; i < parts; ++i) sum += partial[static_cast<size_t>(i) * cols + c];
  out[c] = __float2bfloat16_rn(sum);
}

}  // namespace

// Row ranges a matrix of this shape is cut into, at least 64 rows each: as many CTAs as are resident on 148 SMs, in one wave.
extern "C" int kb_col_sum_parts(int rows, int cols) {
  const int blocks = (cols + COLS - 1) / COLS;
  int parts = CTAS * 148 / blocks;
  if (parts > (rows + 63) / 64) parts = (rows + 63) / 64;
  return parts < 1 ? 1 : parts;
}

extern "C" int kb_col_sum(const void* x, int rows, int cols, float* partial, void* out, void* stream_v) {
  if (rows < 1 || cols < 8 || cols % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) != 0) {
    kb::set_error("kb_col_sum: need rows > 0, columns a multiple of 8 and a 16-byte aligned matrix (got %d x %d)", rows, cols);
    return KB_ERR_ARG;
  }
  const int parts = kb_col_sum_parts(rows, cols);
  if (parts > 1 && partial == nullptr) {
    kb::set_error("kb_col_sum: %d row ranges need a partial buffer", parts);
    return KB_ERR_ARG;
  }
  const int rows_per = (rows + parts - 1) / parts;
  const dim3 grid((cols + COLS - 1) / COLS, parts);
  KB_CUDA_OK(kb::launch_after(col_sum_kernel, grid, 32 * WARPS, stream_v, static_cast<const __nv_bfloat16*>(x), rows, cols, rows_per,
                              parts > 1 ? partial : nullptr, static_cast<__nv_bfloat16*>(out)));
  if (parts > 1) {
    KB_CUDA_OK(kb::launch_after(col_sum_finish_kernel, (cols + 255) / 256, 256, stream_v, static_cast<const float*>(partial), parts, cols,
                                static_cast<__nv_bfloat16*>(out)));
  }
  return KB_OK;
}
