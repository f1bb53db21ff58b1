// Host helpers shared by the launchers of the single-GPU tcgen05 GEMM family.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../common/host_util.h"
#include "gemm_local.cuh"

namespace kbl {

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// bf16 tensor [d2][d1][d0], contiguous, d0 innermost.
inline int make_tmap3(CUtensorMap* map, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t box0, uint32_t box1) {
  static auto encode = KB_DRV(cuTensorMapEncodeTiled);
  if (encode == nullptr) return KB_ERR_UNSUPPORTED;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {d0 * 2, d0 * d1 * 2};
  cuuint32_t box[3] = {box0, box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = kb::with_context([&] {
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) {
    kb::set_error("cuTensorMapEncodeTiled failed: CUresult %d (ptr %p dims %llu %llu %llu)", (int)r, ptr, (unsigned long long)d0,
                  (unsigned long long)d1, (unsigned long long)d2);
    return KB_ERR_CUDA;
  }
  return KB_OK;
}

// bf16 tensor [d2][d1][d0], d0 a multiple of 64, seen as [d2][d0 / 64][d1][64]: a box is `blocks` blocks of 64 elements
// by `box1` rows, in shared memory block by block.
inline int make_tmap4_blocks(CUtensorMap* map, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t box1, uint32_t blocks) {
  static auto encode = KB_DRV(cuTensorMapEncodeTiled);
  if (encode == nullptr) return KB_ERR_UNSUPPORTED;
  cuuint64_t dims[4] = {64, d1, d0 / 64, d2};
  cuuint64_t strides[3] = {d0 * 2, 128, d0 * d1 * 2};
  cuuint32_t box[4] = {64, box1, blocks, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = kb::with_context([&] {
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) {
    kb::set_error("cuTensorMapEncodeTiled failed: CUresult %d (ptr %p dims %llu %llu %llu)", (int)r, ptr, (unsigned long long)d0,
                  (unsigned long long)d1, (unsigned long long)d2);
    return KB_ERR_CUDA;
  }
  return KB_OK;
}

// Whether a launch of `grid` CTAs is set up under the end of the previous kernel of the stream.  Without that it starts 2 to 3 us
// after the end of the one before (a launch in order starts on a 2 us grid); 760 dense products back to back, three weights in
// turn, each way.  Two kinds of launch lose by it:
//   clusters of an odd size that fill the chip: placed one by one as SMs fall free they leave some unused.  26 clusters of five
//     (130 CTAs) 23.1 us in order, 32.2 overlapped and 37.0 43.2; 25 of them 29.0 25.7; 45 of three 25.0 25.4, 43 of them 31.4 29.0;
//     clusters of seven (105 CTAs) gain 2 us.
//   a long read of weights by single CTAs in clusters of two on less than 9/10 of the SMs, which then stand closer together:
//     64 clusters 81.7 us in order, 90.7 overlapped (91 x 8088 x 22632), 60 clusters of 198 MB + 13 %, 56 of 525 MB + 15 %;
//     below 160 MB, or on more SMs, the gain is larger (72 clusters of 186 MB - 5 %, 64 of 96 MB - 7 %).
// Over all of them the launch picked here takes 0.2 % more than the better one, 32 of 1236 more than 3 % (in order: 10 %).
inline bool overlaps(int cluster, int split, int grid, int sms, double weight_bytes) {
  if (cluster % 2 != 0) return cluster == 1 || grid * 8ll < sms * 7ll;
  return cluster != 2 || split != 2 || weight_bytes < 160e6 || grid * 10ll >= sms * 9ll;
}

// Whether the first weights are brought into the L2 before the previous launch has ended (prefetch_weights): dense products of few
// rows, bound by the weights' way from memory, which is idle from that launch's last loads to this one's first.  us, without and
// with, back to back, three weights in turn:
//   1 x 8192 x 8192  26.9  25.0    16 x 7168 x 18432  46.0  44.3    64 x 7168 x 18432  46.6  45.2    128 x 4096 x 4096  13.1  12.3
// Not where `early` fills the ring itself by then, nor from more rows on, whose tensor work it only disturbs: an MLP of 256 tokens
// 72.7 us without and 73.1 with, MoE layers of 32 tokens 94.0 and 94.5; nor for weights along N, which are 256 bytes of each of
// many rows: 24 to 60 MB 5 % longer with it on average (7 x 3376 x 5792 10.8 us without, 11.9 with), 60 to 100 MB 2 %, more than
// that 1 %.  Nor for weights of up to 33 MB, of which the L2 holds four: weights that are there already take 4 to 7 % longer with it,
// others gain the less the smaller they are.  us, one weight again and again, and eight in turn, without and with:
//   16 x 2336 x 5544 (26 MB)  7.9 8.5   9.5  9.2    73 x 9200 x 1632 (30 MB)  8.5 9.1  10.6 10.1    8 x 4096 x 4096 (34 MB)  7.4 7.8  10.1 9.6
//   16 x 4608 x 4608 (42 MB)  8.4 8.8  11.6 10.3    32 x 7168 x 4096 (59 MB) 10.0 10.4 14.2 12.8
inline bool prefetches(const KbLocalGemmArgs& a) {
  return a.kind == KB_LOCAL_DENSE && !a.b_mn && a.M <= 128 && a.early == 0 && 2.0 * a.N * a.K >= 33e6;
}

// One CTA per SM with all of its shared memory, in clusters of `cluster` CTAs.
inline int launch_clusters(const void* fn, int grid, int threads, int cluster, bool overlapped, void* params, void* stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = SMEM_MAX;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (cluster > 1) {
    cudaLaunchAttribute& dim = attr[cfg.numAttrs++];
    dim.id = cudaLaunchAttributeClusterDimension;
    dim.val.clusterDim.x = cluster;
    dim.val.clusterDim.y = 1;
    dim.val.clusterDim.z = 1;
  }
  if (overlapped) attr[cfg.numAttrs++] = kb::overlap_launch();
  void* args[] = {params};
  KB_CUDA_OK(cudaLaunchKernelExC(&cfg, fn, args));
  return KB_OK;
}

}  // namespace kbl
