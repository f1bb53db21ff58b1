// Device code of the single-GPU tcgen05 GEMM family (host side: gemm_local.cu).
//
// One persistent, warp-specialised kernel template covers the products whose
// operands are all on this GPU:
//
//   dense     out[M,N]      = A[M,K] * B[N,K]^T
//   rows      rows of A are grouped (one group per expert); group e is multiplied by its own B[e][N,K]
//   contract  the contraction is grouped: out[e][M,N] = A[rows of e]^T * B[rows of e] (weight gradients)
//
// Each operand is either contiguous along K or along its own M / N dimension: a
// gradient product reads the tensor the forward pass left in memory instead of a
// transposed copy of it.  TMA brings 64-element (128-byte) wide boxes with the
// 128-byte swizzle in both cases; only the box shape and the shared-memory
// descriptors of the MMA differ.
//
// Warp 0 is the TMA producer, warp 1 the MMA issuer, warp 2 owns the TMEM
// allocation, warps 4 to 7 are the epilogue.  Two 256-column accumulators: the
// epilogue of a tile runs under the mainloop of the next one.
//
// A tile has 128 rows (one CTA) or 256 rows (CTA pair, cta_group::2) and `bn`
// columns, a runtime multiple of 32 up to 256: what the launcher picks so that
// the tiles fill the chip (see choose_config in gemm_local.cu).
//
// Split contraction (dense, few tiles): `split` CTAs (or pairs) form one cluster
// and share a tile, each with its part of K.  The fp32 partial tiles are exchanged
// through distributed shared memory (the operand ring is free by then): every
// member owns a part of the tile's columns, receives the other members' partials of
// it and adds them in ascending member order, so the result does not depend on
// timing, and no global workspace, counter or second launch is needed.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../include/kb200.h"

namespace kbl {

using bf16 = __nv_bfloat16;

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int ACC_COLS = 256;  // TMEM columns of one accumulator
constexpr int TMEM_COLS = 512;
constexpr int THREADS = 256;
constexpr int MAX_STAGES = 12;
constexpr int MAX_GROUPS = 1024;
constexpr int BOX_ROWS = 32;
constexpr int EPI_WARP_BYTES = 8192;  // two staging boxes of 32 rows x up to 64 columns
constexpr int EPI_BYTES = 4 * EPI_WARP_BYTES;
constexpr int BAR_BYTES = 256;
constexpr int MN_BLOCK_BYTES = BK * 128;  // M/N-contiguous operand: one box of 64 k rows x 64 elements
constexpr int SMEM_MAX = 232448;
constexpr int CHUNK_COLS = 32;            // split: columns are exchanged in chunks of 32

enum Kind { DENSE = 0, ROWS = 1, CONTRACT = 2 };
enum Act { ACT_NONE = 0, ACT_GELU = 1, ACT_RELU = 2, ACT_SILU = 3 };

struct alignas(64) Params {
  CUtensorMap tmA, tmB, tmOut, tmPre;
  int M, N, K;
  int MBQ, NB, KB;   // scheduling blocks (128 or 256 rows), column blocks, k blocks of the whole contraction
  int bn;            // tile columns
  int group;         // scheduling blocks swept together (rasterisation)
  int groups;
  int split;         // members of a cluster that share a tile
  int stages, a_slot, b_slot;  // operand ring: bytes per stage
  int a_rows;        // rows of A a stage brings in (128 per half, or fewer when M or the groups are smaller)
  int box_cols;      // columns of an output box: 64, or 32 when bn is an odd multiple of 32
  int act;           // applied to the rounded result, or, with pre_in, its derivative at pre_in
  const bf16* bias;
  float bias_scale;
  bf16* out;
  bf16* pre_out;       // value before the activation, or null
  const bf16* pre_in;  // saved value before the activation (backward), or null
  const int32_t* row_start;  // [groups] first row of a group
  const int32_t* row_count;  // [groups]
  uint32_t* status;
  uint64_t limit_ns;
  int timing;  // status[7] receives the microseconds until the last epilogue ended
};

enum Site : uint32_t { SITE_EMPTY = 31, SITE_FULL = 32, SITE_TEMPTY = 33, SITE_TFULL = 34 };

struct Tile {
  int group;    // B / output group
  int row0;     // first row of this CTA's share in A and in the output
  int row_end;  // one past the last valid row
  int n0;       // first column
  int k_row;    // contract: first k row
  int kb;       // k blocks
};

__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(kb::pack_bf16x2(f[0], f[1]), kb::pack_bf16x2(f[2], f[3]), kb::pack_bf16x2(f[4], f[5]), kb::pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  float2 t;
  t = kb::unpack_bf16x2(v.x); f[0] = t.x; f[1] = t.y;
  t = kb::unpack_bf16x2(v.y); f[2] = t.x; f[3] = t.y;
  t = kb::unpack_bf16x2(v.z); f[4] = t.x; f[5] = t.y;
  t = kb::unpack_bf16x2(v.w); f[6] = t.x; f[7] = t.y;
}

__device__ __forceinline__ float sigmoid(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
// tanh form of GELU: x * sigmoid(2u), u = sqrt(2/pi) * (x + 0.044715 x^3)
constexpr float GELU_C = 2.0f * 0.7978845608028654f;
constexpr float GELU_A = 0.044715f;
__device__ __forceinline__ float act_value(int act, float x) {
  if (act == ACT_GELU) return x * sigmoid(GELU_C * x * (1.0f + GELU_A * x * x));
  if (act == ACT_SILU) return x * sigmoid(x);
  return x < 0.0f ? 0.0f : x;
}
__device__ __forceinline__ float act_slope(int act, float x) {
  if (act == ACT_GELU) {
    const float s = sigmoid(GELU_C * x * (1.0f + GELU_A * x * x));
    return s + x * s * (1.0f - s) * GELU_C * (1.0f + 3.0f * GELU_A * x * x);
  }
  if (act == ACT_SILU) {
    const float s = sigmoid(x);
    return s * (1.0f + x * (1.0f - s));
  }
  return x > 0.0f ? 1.0f : 0.0f;
}

// Eight accumulator values of one row -> bf16: (+ bias, one rounding), then the
// activation of the rounded value, or the product with the slope at `pre_in`.
struct Out8 {
  uint4 out, pre;
};
__device__ __forceinline__ Out8 finish8(const Params& p, const float* acc, int row, int col, bool live) {
  float f[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] = acc[e];
  if (p.bias != nullptr && col < p.N) {
    float b[8];
    unpack8(*reinterpret_cast<const uint4*>(p.bias + col), b);  // the same 16 bytes for every lane
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] += p.bias_scale * b[e];
  }
  Out8 o;
  if (p.pre_in != nullptr) {
    float s[8];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (live) v = *reinterpret_cast<const uint4*>(p.pre_in + static_cast<size_t>(row) * p.N + col);
    unpack8(v, s);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= act_slope(p.act, s[e]);
    o.out = pack8(f);
    return o;
  }
  o.pre = pack8(f);
  o.out = o.pre;
  if (p.act != ACT_NONE) {
    float s[8];
    unpack8(o.pre, s);
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = act_value(p.act, s[e]);
    o.out = pack8(s);
  }
  return o;
}

// Shared-memory descriptor of an M/N-contiguous operand with the 128-byte swizzle:
// blocks of 64 elements x 64 k rows (one TMA box, 8 KB), next block MN_BLOCK_BYTES
// further (leading offset), next eight k rows 1024 bytes further (stride offset).
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(MN_BLOCK_BYTES >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// kHalves: 128-row blocks per CTA and tile.  2 (pairs only): a 512-row tile whose two
// halves fill both accumulators.
template <Kind kKind, bool kPair, bool kAMn, bool kBMn, int kHalves>
__global__ void __launch_bounds__(THREADS, 1) gemm_local_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sm_a = base;
  uint8_t* sm_b = sm_a + p.stages * p.a_slot;
  uint8_t* sm_epi = sm_b + p.stages * p.b_slot;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm_epi + EPI_BYTES);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= BAR_BYTES, "barrier block too small");
  int32_t* pref = reinterpret_cast<int32_t*>(sm_epi + EPI_BYTES + BAR_BYTES);  // [groups + 1] row blocks before a group
  int32_t* g_start = pref + p.groups + 1;                                      // [groups]
  int32_t* g_count = g_start + p.groups;                                       // [groups]

  const uint64_t t_start = p.timing ? kb::globaltimer_ns() : 0;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t ctarank = (kPair || p.split > 1) ? kb::cluster_ctarank() : 0u;
  const uint32_t half = kPair ? (ctarank & 1u) : 0u;       // which 128 rows of a pair's tile
  const uint32_t lead = kPair ? (ctarank & ~1u) : ctarank;  // cluster rank of the CTA that issues the MMAs
  const bool leader = half == 0u;
  const int member = static_cast<int>(kPair ? (ctarank >> 1) : ctarank);  // part of K this CTA (pair) works on when split > 1
  const int cta_per_tile = (kPair ? 2 : 1) * p.split;
  const int sched_id = static_cast<int>(blockIdx.x) / cta_per_tile;
  const int sched_n = static_cast<int>(gridDim.x) / cta_per_tile;
  constexpr int CTA_ROWS = kHalves * BM;
  constexpr int TILE_ROWS = kPair ? 2 * CTA_ROWS : CTA_ROWS;
  // rows of one scheduling block: groups with few rows get low tiles (one CTA, 32 or 64 of the MMA's 128 rows)
  const int block_rows = (kKind == ROWS && !kPair) ? p.a_rows : TILE_ROWS;
  const int b_cols = kPair ? p.bn / 2 : p.bn;  // columns of B this CTA stages

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      kb::mbar_init(&full[s], 1);
      kb::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      kb::mbar_init(&tfull[a], 1);
      kb::mbar_init(&tempty[a], kPair ? 8 : 4);
    }
    *abort_flag = 0;
    kb::mbar_fence_init();
  }
  if (warp == 2) {
    if constexpr (kPair) {
      kb::tmem_alloc_pair(tmem_slot, TMEM_COLS);
      kb::tmem_relinquish_pair();
    } else {
      kb::tmem_alloc(tmem_slot, TMEM_COLS);
      kb::tmem_relinquish();
    }
  }
  if (warp == 3 && lane == 0) {
    kb::tma_prefetch_desc(&p.tmA);
    kb::tma_prefetch_desc(&p.tmB);
    kb::tma_prefetch_desc(&p.tmOut);
  }
  if constexpr (kKind != DENSE) {
    for (int e = tid; e < p.groups; e += THREADS) {
      g_start[e] = p.row_start[e];
      g_count[e] = p.row_count[e];
    }
    if constexpr (kKind == ROWS) {
      __syncthreads();
      if (warp == 0) {  // exclusive prefix of the groups' row blocks
        int carry = 0;
        for (int e0 = 0; e0 < p.groups; e0 += 32) {
          const int e = e0 + lane;
          int v = e < p.groups ? (g_count[e] + block_rows - 1) / block_rows : 0;
          const int mine = v;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += n;
          }
          if (e < p.groups) pref[e] = carry + v - mine;
          carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) pref[p.groups] = carry;
      }
    }
  }
  kb::tc_fence_before_sync();
  __syncthreads();
  if (kPair || p.split > 1) kb::cluster_sync_all();  // the other CTAs' barriers exist before anything signals them
  kb::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int total_tiles = kKind == DENSE ? p.MBQ * p.NB : kKind == ROWS ? pref[p.groups] * p.NB : p.groups * p.MBQ * p.NB;

  // Position in the static schedule -> tile.  Dense: groups of `group` row blocks
  // are swept column by column, so that the tiles in flight share few panels of A
  // and B.  Grouped: group by group; inside a group the row blocks of a column
  // block follow each other, they share the group's B panel.
  auto tile_at = [&](int pos) -> Tile {
    Tile t;
    int mbq, nb;
    t.k_row = 0;
    t.kb = p.KB;
    if constexpr (kKind == DENSE) {
      const int per_group = p.group * p.NB;
      const int g = pos / per_group;
      const int r = pos - g * per_group;
      const int gs = min(p.MBQ - g * p.group, p.group);
      nb = r / gs;
      mbq = g * p.group + (r - nb * gs);
      t.group = 0;
      t.row0 = mbq * TILE_ROWS + static_cast<int>(half) * CTA_ROWS;
      t.row_end = p.M;
    } else if constexpr (kKind == ROWS) {
      const int block = pos / p.NB;  // counts row blocks: group e holds blocks pref[e] .. pref[e + 1] - 1
      int lo = 0, hi = p.groups - 1;
      while (lo < hi) {  // last group with pref <= block: it is not empty
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= block) lo = mid;
        else hi = mid - 1;
      }
      const int blocks = pref[lo + 1] - pref[lo];
      const int r = pos - pref[lo] * p.NB;
      nb = r / blocks;
      mbq = r - nb * blocks;
      t.group = lo;
      t.row0 = g_start[lo] + mbq * block_rows + static_cast<int>(half) * CTA_ROWS;
      t.row_end = min(g_start[lo] + g_count[lo], t.row0 + (kPair ? CTA_ROWS : block_rows));
    } else {
      const int per = p.MBQ * p.NB;
      t.group = pos / per;
      const int r = pos - t.group * per;
      nb = r / p.MBQ;
      mbq = r - nb * p.MBQ;
      t.row0 = mbq * TILE_ROWS + static_cast<int>(half) * CTA_ROWS;
      t.row_end = p.M;
      t.k_row = g_start[t.group];
      t.kb = (g_count[t.group] + BK - 1) / BK;
    }
    t.n0 = nb * p.bn;
    return t;
  };
  // k blocks [k0, k1) of a tile that this member works on
  auto k_range = [&](const Tile& t, int& k0, int& k1) {
    k0 = static_cast<int>(static_cast<long long>(t.kb) * member / p.split);
    k1 = static_cast<int>(static_cast<long long>(t.kb) * (member + 1) / p.split);
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer ----
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      const uint32_t a_bytes = static_cast<uint32_t>(p.a_rows) * BK * 2;
      const uint32_t stage_bytes = a_bytes + static_cast<uint32_t>(b_cols) * BK * 2;
      for (int pos = sched_id; ok && pos < total_tiles; pos += sched_n) {
        const Tile t = tile_at(pos);
        int k0, k1;
        k_range(t, k0, k1);
        const int bz = kKind == ROWS ? t.group : 0;
        const int nrow = t.n0 + static_cast<int>(half) * b_cols;
        for (int k = k0; k < k1; ++k) {
          if (!kb::mbar_wait_bounded(&empty[s], ph ^ 1u, p.limit_ns, 400)) {
            kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_EMPTY, (uint32_t)pos, 0);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* da = sm_a + s * p.a_slot;
          uint8_t* db = sm_b + s * p.b_slot;
          uint32_t bar = kb::smem_u32(&full[s]);
          if constexpr (kPair) {
            if (leader) kb::mbar_arrive_expect_tx(&full[s], 2 * stage_bytes);
            bar = kb::map_to_cta(bar, lead);  // both CTAs' bytes are counted on the leader's barrier
          } else {
            kb::mbar_arrive_expect_tx(&full[s], stage_bytes);
          }
          if constexpr (kAMn) {
#pragma unroll
            for (int i = 0; i < CTA_ROWS / 64; ++i) {
              kb::tma_load_3d<kPair>(da + i * MN_BLOCK_BYTES, &p.tmA, bar, t.row0 + i * 64, t.k_row + k * BK, 0);
            }
          } else {
            kb::tma_load_3d<kPair>(da, &p.tmA, bar, k * BK, t.row0, 0);
          }
          if constexpr (kBMn) {
            for (int i = 0; i < b_cols / 64; ++i) {
              kb::tma_load_3d<kPair>(db + i * MN_BLOCK_BYTES, &p.tmB, bar, nrow + i * 64, t.k_row + k * BK, bz);
            }
          } else {
            kb::tma_load_3d<kPair>(db, &p.tmB, bar, k * BK, nrow, bz);
          }
          if (++s == p.stages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer ----
    // The whole warp walks the loop, one elected lane issues (see umma_f16_x4).
    if (leader) {
      const uint32_t idesc = kb::umma_idesc_bf16(kPair ? 2 * BM : BM, p.bn) | (kAMn ? 1u << 15 : 0u) | (kBMn ? 1u << 16 : 0u);
      // one K step: 16 elements of a 128-byte row, or 16 of the k rows
      constexpr uint32_t A_STEP = (kAMn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      constexpr uint32_t B_STEP = (kBMn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      const uint64_t da = kAMn ? desc_mn_sw128(kb::smem_u32(sm_a)) : kb::umma_desc_k_sw128(kb::smem_u32(sm_a));
      const uint64_t db = kBMn ? desc_mn_sw128(kb::smem_u32(sm_b)) : kb::umma_desc_k_sw128(kb::smem_u32(sm_b));
      const uint32_t a_lo = static_cast<uint32_t>(da), a_hi = static_cast<uint32_t>(da >> 32);
      const uint32_t b_lo = static_cast<uint32_t>(db), b_hi = static_cast<uint32_t>(db >> 32);
      const uint32_t a_inc = static_cast<uint32_t>(p.a_slot) >> 4, b_inc = static_cast<uint32_t>(p.b_slot) >> 4;
      const uint32_t empty0 = kPair ? kb::map_to_cta(kb::smem_u32(empty), lead) : kb::smem_u32(empty);
      const uint32_t empty1 = kPair ? kb::map_to_cta(kb::smem_u32(empty), lead + 1u) : 0u;
      uint32_t s = 0;
      uint32_t ph = 0;
      uint32_t it = 0;
      bool ok = true;
      for (int pos = sched_id; ok && pos < total_tiles; pos += sched_n, ++it) {
        const Tile t = tile_at(pos);
        int k0, k1;
        k_range(t, k0, k1);
        for (int k = k0; k < k1 || k == k0; ++k) {
          const bool work = k < k1;  // an empty group still hands its accumulator on
          if (work && ok && !kb::mbar_wait_bounded(&full[s], ph, p.limit_ns)) {
            kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_FULL, (uint32_t)pos, 0);
            ok = false;
          }
#pragma unroll
          for (int h = 0; h < kHalves; ++h) {
            // one half: accumulators alternate from tile to tile; two halves: a tile fills both
            const uint32_t acc = kHalves == 2 ? static_cast<uint32_t>(h) : it & 1u;
            const uint32_t use = kHalves == 2 ? it : it >> 1;
            if (k == k0) {
              if (ok && !kb::mbar_wait_bounded(&tempty[acc], (use & 1u) ^ 1u, p.limit_ns)) {
                kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_TEMPTY, (uint32_t)pos, 0);
                ok = false;
              }
            }
            if (!ok) break;
            kb::tc_fence_after_sync();
            if (work) {
              kb::umma_f16_x4<kPair>(tmem_base + acc * ACC_COLS, a_lo + s * a_inc + h * (BM * BK * 2 / 16), a_hi, b_lo + s * b_inc, b_hi,
                                     A_STEP, B_STEP, idesc, k != k0 ? 1u : 0u);
            }
            if (k + 1 >= k1) {
              const uint32_t f = kb::smem_u32(&tfull[acc]);
              kb::umma_commit_warp<kPair>(kPair ? kb::map_to_cta(f, lead) : f);
              if constexpr (kPair) kb::umma_commit_warp<kPair>(kb::map_to_cta(f, lead + 1u));
            }
          }
          if (!ok) {
            *abort_flag = 1;
            break;
          }
          if (!work) break;
          // the stage is free (in both CTAs of a pair) once these MMAs have read it
          kb::umma_commit_warp<kPair>(empty0 + s * 8);
          if constexpr (kPair) kb::umma_commit_warp<kPair>(empty1 + s * 8);
          if (++s == static_cast<uint32_t>(p.stages)) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4 && p.split == 1) {
    // ---------------------------------------------------------- epilogue ----
    const int q = warp - 4;
    uint8_t* warp_epi = sm_epi + q * EPI_WARP_BYTES;
    uint32_t it = 0;
    int box = 0;  // next staging box
    for (int pos = sched_id; pos < total_tiles; pos += sched_n, ++it) {
      const Tile t = tile_at(pos);
#pragma unroll 1
      for (int hb = 0; hb < kHalves; ++hb) {
      const uint32_t acc = kHalves == 2 ? static_cast<uint32_t>(hb) : it & 1u;
      const uint32_t aph = (kHalves == 2 ? it : it >> 1) & 1u;
      if (*abort_flag == 0 && !kb::mbar_wait_bounded(&tfull[acc], aph, p.limit_ns, 2000)) {
        kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_TFULL, (uint32_t)pos, 0);
        *abort_flag = 1;
      }
      kb::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * ACC_COLS;
      const int gr0 = t.row0 + hb * BM + q * 32;
      const int row = gr0 + lane;
      const bool row_ok = row < t.row_end;
      // A box leaves through TMA unless it would reach into the next group's rows.
      const bool tma_ok = kKind != ROWS || gr0 + BOX_ROWS <= t.row_end;
      const int cols = min(p.bn, p.N - t.n0);
      const int oz = kKind == CONTRACT ? t.group : 0;
      if (gr0 < t.row_end) {
#pragma unroll 1
        for (int c = 0; c < cols; c += p.box_cols) {
          const int col0 = t.n0 + c;
          uint8_t* box_out = warp_epi + box * (EPI_WARP_BYTES / 2);
          uint8_t* box_pre = warp_epi + (box ^ 1) * (EPI_WARP_BYTES / 2);
          if (tma_ok) {  // the stores that last read the box(es) have finished reading
            if (lane == 0) {
              if (p.pre_out != nullptr) kb::bulk_wait_group_read<0>();
              else kb::bulk_wait_group_read<1>();
            }
            __syncwarp();
          }
#pragma unroll 1
          for (int h = 0; h < p.box_cols; h += 32) {
            uint32_t r[32];
            if (kKind == CONTRACT && t.kb == 0) {  // an empty group: nothing was accumulated
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            } else {
              kb::tmem_ld_32x32(taddr + c + h, r);
              kb::tmem_ld_wait();
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int col = col0 + h + 8 * i;
              const Out8 o = finish8(p, reinterpret_cast<const float*>(r) + 8 * i, row, col, row_ok && col < p.N);
              if (tma_ok) {
                // 16-byte chunk j of the row at position j ^ (row & 7) of its 128 bytes (64-byte rows: j ^ ((row / 2) & 3))
                const int j = h / 8 + i;
                const int at = p.box_cols == 64 ? lane * 128 + ((j ^ (lane & 7)) * 16) : lane * 64 + ((j ^ ((lane >> 1) & 3)) * 16);
                *reinterpret_cast<uint4*>(box_out + at) = o.out;
                if (p.pre_out != nullptr) *reinterpret_cast<uint4*>(box_pre + at) = o.pre;
              } else if (row_ok && col < p.N) {
                const size_t at = static_cast<size_t>(row) * p.N + col;
                *reinterpret_cast<uint4*>(p.out + at) = o.out;
                if (p.pre_out != nullptr) *reinterpret_cast<uint4*>(p.pre_out + at) = o.pre;
              }
            }
          }
          if (tma_ok) {
            kb::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              kb::tma_store_3d(&p.tmOut, box_out, col0, gr0, oz);
              if (p.pre_out != nullptr) kb::tma_store_3d(&p.tmPre, box_pre, col0, gr0, oz);
              kb::bulk_commit_group();
            }
            box ^= 1;
          }
        }
      }
      kb::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kPair) {
          if (leader) kb::mbar_arrive(&tempty[acc]);
          else kb::mbar_arrive_cluster(kb::map_to_cta(kb::smem_u32(&tempty[acc]), lead));
        } else {
          kb::mbar_arrive(&tempty[acc]);
        }
      }
      }
    }
    if (lane == 0) kb::bulk_wait_group<0>();  // the boxes are read and the output is written before the CTA leaves
  } else if (warp == 4 && p.split > 1) {
    // The members of a cluster work on one tile each: wait here until this CTA's partial is complete.
    if (!kb::mbar_wait_bounded(&tfull[0], 0u, p.limit_ns, 1000)) {
      kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_TFULL, (uint32_t)sched_id, 0);
      *abort_flag = 1;
    }
    kb::tc_fence_before_sync();
  }

  if constexpr (kKind == DENSE) {
    if (p.split > 1) {
      // ------------------------------------------- exchange of the partials ----
      // Chunk c of 32 columns belongs to member c * split / chunks.  Slot (chunk,
      // source) of the owner's operand ring holds 128 rows x 32 columns as
      // [4-column group][row] float4: neighbouring lanes write neighbouring 16 bytes.
      __syncthreads();
      kb::cluster_sync_all();  // every member's MMAs have finished: all operand rings are free
      kb::tc_fence_after_sync();
      const Tile t = tile_at(sched_id);
      const int chunks = p.bn / CHUNK_COLS;
      const int q = warp & 3;            // TMEM lane quadrant of this warp
      const int gr0 = t.row0 + q * 32;
      const int row = gr0 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      constexpr int SLOT = BM * CHUNK_COLS * 4;
      const bool live = gr0 < t.row_end;
      if (live) {
        for (int c = warp >> 2; c < chunks; c += 2) {
          const int owner = c * p.split / chunks;
          if (owner == member || t.n0 + c * CHUNK_COLS >= p.N) continue;
          const int first = (owner * chunks + p.split - 1) / p.split;  // the owner's first chunk
          const int src = member < owner ? member : member - 1;
          uint32_t r[32];
          kb::tmem_ld_32x32(taddr + c * CHUNK_COLS, r);
          kb::tmem_ld_wait();
          const uint32_t to = kb::map_to_cta(kb::smem_u32(base + ((c - first) * (p.split - 1) + src) * SLOT),
                                             static_cast<uint32_t>(owner) * (kPair ? 2u : 1u) + half);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            kb::st_shared_cluster_v4(to + (i * BM + q * 32 + lane) * 16, r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
          }
        }
      }
      kb::cluster_sync_all();  // the partials are in place
      if (live) {
        for (int c = warp >> 2; c < chunks; c += 2) {
          const int col0 = t.n0 + c * CHUNK_COLS;
          if (c * p.split / chunks != member || col0 >= p.N) continue;
          const int first = (member * chunks + p.split - 1) / p.split;
          uint32_t r[32];
          kb::tmem_ld_32x32(taddr + c * CHUNK_COLS, r);
          kb::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = 0.f;
            for (int m = 0; m < p.split; ++m) {  // ascending member order
              if (m == member) {
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += __uint_as_float(r[8 * i + e]);
                continue;
              }
              const uint8_t* slot = base + ((c - first) * (p.split - 1) + (m < member ? m : m - 1)) * SLOT;
#pragma unroll
              for (int g = 0; g < 2; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(slot + ((2 * i + g) * BM + q * 32 + lane) * 16);
                f[4 * g] += v.x; f[4 * g + 1] += v.y; f[4 * g + 2] += v.z; f[4 * g + 3] += v.w;
              }
            }
            const int col = col0 + 8 * i;
            const bool ok = row < t.row_end && col < p.N;
            const Out8 o = finish8(p, f, row, col, ok);
            if (ok) {
              const size_t at = static_cast<size_t>(row) * p.N + col;
              *reinterpret_cast<uint4*>(p.out + at) = o.out;
              if (p.pre_out != nullptr) *reinterpret_cast<uint4*>(p.pre_out + at) = o.pre;
            }
          }
        }
      }
    }
  }

  if (p.timing && p.status != nullptr && warp == 4 && lane == 0) {
    atomicMax(&p.status[7], static_cast<uint32_t>((kb::globaltimer_ns() - t_start) / 1000));
  }
  kb::tc_fence_before_sync();
  __syncthreads();
  if constexpr (kPair) kb::cluster_sync_all();  // nobody leaves while the partner may still signal or read
  if (warp == 2) {
    kb::tc_fence_after_sync();
    if constexpr (kPair) kb::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else kb::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace kbl
