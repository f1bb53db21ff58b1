// Host side of the single-GPU tcgen05 GEMM family (device code: gemm_local.cuh).
#include "gemm_local.cuh"

#include <stdlib.h>
#include <string.h>

namespace {

using namespace kbl;

// bf16 tensor [d2][d1][d0], contiguous, d0 innermost.
int make_tmap3(CUtensorMap* map, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t box0, uint32_t box1, bool swizzle64) {
  static auto encode = KB_DRV(cuTensorMapEncodeTiled);
  if (encode == nullptr) return KB_ERR_UNSUPPORTED;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {d0 * 2, d0 * d1 * 2};
  cuuint32_t box[3] = {box0, box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    kb::set_error("cuTensorMapEncodeTiled failed: CUresult %d (ptr %p dims %llu %llu %llu)", (int)r, ptr, (unsigned long long)d0,
                  (unsigned long long)d1, (unsigned long long)d2);
    return KB_ERR_CUDA;
  }
  return KB_OK;
}

// Environment switches, read once per process.
struct Env {
  bool no_pair, timing;
  Env() {
    const char* v = getenv("KB200_GEMM_NO_PAIR");
    no_pair = v != nullptr && v[0] == '1';
    v = getenv("KB200_GEMM_TIMING");
    timing = v != nullptr && v[0] == '1';
  }
};
const Env& env() {
  static const Env e;
  return e;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

struct Config {
  bool pair;
  int bn, split;
  bool tall = false;  // pair with 256 rows per CTA
};

// Columns a tile may have: multiples of 32; an operand that is contiguous along N
// comes in boxes of 64 columns per CTA.
bool bn_ok(int bn, bool pair, bool b_mn) {
  const int per_cta = pair ? bn / 2 : bn;
  return b_mn ? per_cta % 64 == 0 : bn % 32 == 0;
}

Config choose_config(int M, int N, int K, bool a_mn, bool b_mn, int sms, int shape) {
  (void)a_mn;
  Config best = {false, 256, 1};
  double best_t = 1e30;
  const int KB = ceil_div(K, BK);
  for (int s = 0; s < 3; ++s) {
    if (shape >= 0 ? s != shape : s != 0 && M <= 128) continue;
    const bool pair = s > 0, tall = s == 2;
    const int units = pair ? sms / 2 : sms;
    for (int bn = 64; bn <= 256; bn += 32) {
      if (!bn_ok(bn, pair, b_mn) || (tall && bn != 256)) continue;
      const int tiles = ceil_div(M, 128 << s) * ceil_div(N, bn);
      for (int split = 1; split <= (tall ? 1 : pair ? 4 : 8); ++split) {
        if (split > 1 && (tiles * split > units || KB < 4 * split)) break;
        const int waves = ceil_div(tiles * split, units);
        const double kb_ns = (tall ? 2 : 1) * (290.0 * (bn < 96 ? 96 : bn) / 256.0 + (pair ? 0 : 20));
        const double t = waves * (ceil_div(KB, split) * kb_ns) + 1500.0 + (split > 1 ? 2500.0 : 0.0);
        if (t < best_t) {
          best_t = t;
          best = {pair, bn, split, tall};
        }
      }
    }
  }
  return best;
}

int device_info(int* dev_out, int* sms_out) {
  static int cached_sms[64] = {0};
  int dev = 0, sms = 0;
  KB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && cached_sms[dev] > 0) {
    sms = cached_sms[dev];
  } else {
    KB_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (dev >= 0 && dev < 64) cached_sms[dev] = sms;
  }
  *dev_out = dev;
  *sms_out = sms;
  return KB_OK;
}

template <Kind kKind, bool kAMn, bool kBMn>
const void* kernel_of(const Config& c) {
  if constexpr (kKind == DENSE) {
    if (c.tall) return (const void*)gemm_local_kernel<kKind, true, kAMn, kBMn, 2>;
  }
  return c.pair ? (const void*)gemm_local_kernel<kKind, true, kAMn, kBMn, 1> : (const void*)gemm_local_kernel<kKind, false, kAMn, kBMn, 1>;
}

}  // namespace

extern "C" int kb_gemm_local_config(int M, int N, int K, int b_mn, int sms, int* pair, int* bn, int* split) {
  if (M <= 0 || N <= 0 || K <= 0 || sms < 2 || !pair || !bn || !split) return KB_ERR_ARG;
  const Config c = choose_config(M, N, K, false, b_mn != 0, sms, -1);
  *pair = c.tall ? 2 : c.pair ? 1 : 0;
  *bn = c.bn;
  *split = c.split;
  return KB_OK;
}

extern "C" int kb_gemm_local(const KbLocalGemmArgs* a, void* stream_v) {
  if (a == nullptr) return KB_ERR_ARG;
  const bool contract = a->kind == KB_LOCAL_CONTRACT;
  if (a->kind < 0 || a->kind > 2 || a->act < 0 || a->act > 3) {
    kb::set_error("kb_gemm_local: unknown kind %d or activation %d", a->kind, a->act);
    return KB_ERR_ARG;
  }
  const bool a_mn = contract || a->a_mn, b_mn = contract || a->b_mn;
  // TMA rows are multiples of 16 bytes: the contiguous extent of every tensor is a multiple of 8.
  if (a->M <= 0 || a->N <= 0 || a->K <= 0 || a->N % 8 != 0 || (!a_mn && a->K % 8 != 0) || (!b_mn && a->K % 8 != 0) ||
      (a_mn && a->M % 8 != 0)) {
    kb::set_error("kb_gemm_local: need M,N,K > 0 and contiguous extents that are multiples of 8 (got %d %d %d)", a->M, a->N, a->K);
    return KB_ERR_ARG;
  }
  const bool grouped = a->kind != KB_LOCAL_DENSE;
  if (grouped && (a->groups < 1 || a->groups > MAX_GROUPS || a->row_start == nullptr || a->row_count == nullptr || a->bias != nullptr ||
                  (a->kind == KB_LOCAL_ROWS && a_mn))) {
    kb::set_error("kb_gemm_local: bad groups (%d, at most %d, with row tables, without bias)", a->groups, MAX_GROUPS);
    return KB_ERR_ARG;
  }
  if (a->kind == KB_LOCAL_DENSE && a_mn && !b_mn) {
    kb::set_error("kb_gemm_local: A contiguous along M is built only with B contiguous along N");
    return KB_ERR_UNSUPPORTED;
  }
  auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
  if (a->A == nullptr || a->B == nullptr || a->out == nullptr || misaligned(a->A) || misaligned(a->B) || misaligned(a->out) ||
      misaligned(a->bias) || misaligned(a->pre_out) || misaligned(a->pre_in)) {
    kb::set_error("kb_gemm_local: operand pointers must be given and 16-byte aligned");
    return KB_ERR_ARG;
  }
  int dev = 0, sms = 0;
  int rc = device_info(&dev, &sms);
  if (rc != KB_OK) return rc;
  const int cap = a->num_ctas > 0 && a->num_ctas < sms ? a->num_ctas : sms;

  const int groups = grouped ? a->groups : 1;
  int shape = a->pair;  // -1: choose, 0: one CTA, 1: pair, 2: tall pair
  if (cap < 2 || env().no_pair) shape = 0;
  Config c;
  if (a->kind == KB_LOCAL_DENSE) {
    if (shape == 1 && a->M <= 128) shape = 0;  // a pair's second CTA would hold padding only
    c = choose_config(a->M, a->N, a->K, a_mn, b_mn, cap, shape);
  } else {
    // Rows per group decide: with fewer than about 1.5 tiles of 256 rows per group a pair
    // would work mostly on padding.
    const double per_group = contract ? a->M : static_cast<double>(a->M) / groups;
    c.pair = shape < 0 ? per_group >= 384 : shape > 0;
    // few rows per group: the weights are the traffic, narrow tiles spread them evenly over the SMs
    c.bn = a->kind == KB_LOCAL_ROWS && per_group <= 64 ? 64 : a->N <= 64 ? 64 : a->N <= 128 ? 128 : 256;
    c.split = 1;
    if (!bn_ok(c.bn, c.pair, b_mn)) c.bn = 128;
  }
  if (a->bn > 0) c.bn = a->bn;
  if (a->split > 0) c.split = a->split;
  const int KB = ceil_div(a->K, BK);
  if (c.bn < 32 || c.bn > 256 || !bn_ok(c.bn, c.pair, b_mn) || c.split > (c.pair ? 4 : 8) || c.split > KB || ((grouped || c.tall) && c.split > 1)) {
    kb::set_error("kb_gemm_local: tile configuration pair=%d bn=%d split=%d does not fit the problem", c.pair, c.bn, c.split);
    return KB_ERR_ARG;
  }

  Params p;
  memset(&p, 0, sizeof(p));
  p.M = a->M;
  p.N = a->N;
  p.K = a->K;
  // A single CTA whose rows are few brings in only those: the MMA reads 128 rows of
  // shared memory, what lies behind the box only reaches accumulator rows that are not
  // stored.  Groups: 32 or 64 rows per tile when the average group fits it comfortably.
  p.a_rows = c.tall ? 256 : 128;
  if (a->kind == KB_LOCAL_ROWS && !c.pair) {
    const int avg = a->M / groups;
    p.a_rows = avg <= 20 ? 32 : avg <= 48 ? 64 : 128;
  } else if (!c.pair && !a_mn && a->M < 128) {
    p.a_rows = ceil_div(a->M, 8) * 8;
  }
  const int tile_rows = c.tall ? 512 : c.pair ? 256 : a->kind == KB_LOCAL_ROWS ? p.a_rows : 128;
  p.MBQ = ceil_div(a->M, tile_rows);
  p.NB = ceil_div(a->N, c.bn);
  p.KB = KB;
  p.bn = c.bn;
  p.group = (c.tall ? 4096 : 2048) / tile_rows;
  p.groups = grouped ? groups : 0;
  p.split = c.split;
  p.a_slot = p.a_rows * BK * 2;
  p.b_slot = (c.pair ? c.bn / 2 : c.bn) * BK * 2;
  const int tables = grouped ? (3 * groups + 1) * 4 : 4;
  int stages = (SMEM_MAX - 1024 - EPI_BYTES - BAR_BYTES - tables) / (p.a_slot + p.b_slot);
  if (stages > MAX_STAGES) stages = MAX_STAGES;
  p.stages = stages;
  // the last A slot is read up to 128 rows far: the B slots behind it cover that
  if (p.stages < 2 || p.stages * p.b_slot < 16384) {
    kb::set_error("kb_gemm_local: operand ring too small");
    return KB_ERR_ARG;
  }
  if (c.split > 1) {
    const int chunks = c.bn / CHUNK_COLS;
    const int need = ceil_div(chunks, c.split) * (c.split - 1) * BM * CHUNK_COLS * 4;
    if (need > p.stages * (p.a_slot + p.b_slot) + EPI_BYTES) {
      kb::set_error("kb_gemm_local: partial tiles do not fit the operand ring");
      return KB_ERR_ARG;
    }
  }
  p.box_cols = c.bn % 64 == 0 ? 64 : 32;
  p.act = a->act;
  p.bias = static_cast<const bf16*>(a->bias);
  p.bias_scale = a->bias_scale;
  p.out = static_cast<bf16*>(a->out);
  p.pre_out = static_cast<bf16*>(a->pre_out);
  p.pre_in = static_cast<const bf16*>(a->pre_in);
  p.row_start = a->row_start;
  p.row_count = a->row_count;
  p.status = a->status;
  p.limit_ns = a->wait_limit_ns ? a->wait_limit_ns : 2000000000ull;
  p.timing = env().timing ? 1 : 0;

  const uint64_t bz = a->kind == KB_LOCAL_ROWS ? groups : 1, oz = contract ? groups : 1;
  rc = a_mn ? make_tmap3(&p.tmA, a->A, a->M, a->K, 1, 64, BK, false) : make_tmap3(&p.tmA, a->A, a->K, a->M, 1, BK, p.a_rows, false);
  if (rc != KB_OK) return rc;
  rc = b_mn ? make_tmap3(&p.tmB, a->B, a->N, a->K, bz, 64, BK, false)
            : make_tmap3(&p.tmB, a->B, a->K, a->N, bz, BK, c.pair ? c.bn / 2 : c.bn, false);
  if (rc != KB_OK) return rc;
  rc = make_tmap3(&p.tmOut, a->out, a->N, a->M, oz, p.box_cols, BOX_ROWS, p.box_cols == 32);
  if (rc != KB_OK) return rc;
  if (p.pre_out != nullptr) {
    rc = make_tmap3(&p.tmPre, a->pre_out, a->N, a->M, oz, p.box_cols, BOX_ROWS, p.box_cols == 32);
    if (rc != KB_OK) return rc;
  }

  const int cluster = (c.pair ? 2 : 1) * c.split;
  int grid;
  if (c.split > 1) {
    grid = p.MBQ * p.NB * cluster;  // one tile per cluster
  } else {
    grid = c.pair ? cap & ~1 : cap;
    // ROWS: at most one partly filled row block per group on top of the full ones
    const long long blocks = a->kind == KB_LOCAL_ROWS ? a->M / tile_rows + groups : static_cast<long long>(groups) * p.MBQ;
    if (grid > blocks * p.NB * cluster) grid = static_cast<int>(blocks * p.NB * cluster);
  }

  const int variant = a->kind == KB_LOCAL_ROWS ? (b_mn ? 4 : 3) : contract ? 5 : a_mn ? 2 : b_mn ? 1 : 0;
  const void* fn = nullptr;
  switch (variant) {
    case 0: fn = kernel_of<DENSE, false, false>(c); break;
    case 1: fn = kernel_of<DENSE, false, true>(c); break;
    case 2: fn = kernel_of<DENSE, true, true>(c); break;
    case 3: fn = kernel_of<ROWS, false, false>(c); break;
    case 4: fn = kernel_of<ROWS, false, true>(c); break;
    default: fn = kernel_of<CONTRACT, true, true>(c); break;
  }
  const int attr_row = c.tall ? 2 : c.pair ? 1 : 0;
  static bool attr_set[64][3][6] = {};
  if (dev < 0 || dev >= 64 || !attr_set[dev][attr_row][variant]) {
    KB_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    if (dev >= 0 && dev < 64) attr_set[dev][attr_row][variant] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_MAX;
  cfg.stream = static_cast<cudaStream_t>(stream_v);
  cudaLaunchAttribute attr[1];
  if (cluster > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  void* args[] = {&p};
  KB_CUDA_OK(cudaLaunchKernelExC(&cfg, fn, args));
  return KB_OK;
}
