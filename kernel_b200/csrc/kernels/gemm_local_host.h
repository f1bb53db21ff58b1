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
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
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
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    kb::set_error("cuTensorMapEncodeTiled failed: CUresult %d (ptr %p dims %llu %llu %llu)", (int)r, ptr, (unsigned long long)d0,
                  (unsigned long long)d1, (unsigned long long)d2);
    return KB_ERR_CUDA;
  }
  return KB_OK;
}

// Whether a launch of `grid` CTAs is set up under the end of the previous kernel of the stream.  Without that it starts up
// to 2 us after the end of the one before.  Not so where clusters of an odd size fill the chip: placed one by one as SMs
// fall free they leave some unused.  Launched in order and overlapped, us:
//   64 x 7168 x 18432   clusters of 2 on 112 SMs 48.4 46.9   of 4 on 128 49.1 46.9   of 3 on 114 47.9 46.2   of 3 on 135 47.6 50.2
//   256 x 4096 x 14336  clusters of 6 on 132 SMs 32.9 30.2   of 4 on 128 32.9 30.6   of 3 on 114 36.8 35.2   of 3 on 132 34.9 37.0
// Clusters of eight wait longest for SMs that are free together (195 x 3200 x 26136 on 120 SMs costs 1.8 us overlapped).
inline bool overlaps(int cluster, int grid, int sms) { return cluster == 1 || (cluster < 8 && (cluster % 2 == 0 || grid * 100ll < sms * 88ll)); }

// One CTA per SM with all of its shared memory, in clusters of `cluster` CTAs.
inline int launch_clusters(const void* fn, int grid, int threads, int cluster, int sms, void* params, void* stream) {
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
  if (overlaps(cluster, grid, sms)) attr[cfg.numAttrs++] = kb::overlap_launch();
  void* args[] = {params};
  KB_CUDA_OK(cudaLaunchKernelExC(&cfg, fn, args));
  return KB_OK;
}

}  // namespace kbl
