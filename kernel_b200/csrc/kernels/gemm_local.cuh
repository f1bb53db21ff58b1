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
// allocation, warps 4 to 11 are the epilogue.  Two 256-column accumulators: the
// epilogue of a tile runs under the mainloop of the next one.
//
// A tile has 128 rows (one CTA) or 256 rows (CTA pair, cta_group::2) and `bn`
// columns, a runtime multiple of 32 up to 256: what the launcher picks so that
// the tiles fill the chip (see choose_config in gemm_local.cu; choose
// weighs it against exchanged operands, gemm_swap.cuh).
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

#include <type_traits>

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
constexpr int THREADS = 384;
constexpr int EPI_WARPS = 8;  // two per TMEM lane quadrant
constexpr int MAX_STAGES = 12;
constexpr int MAX_GROUPS = 1024;
constexpr int BAR_BYTES = 256;
constexpr int MN_BLOCK_BYTES = BK * 128;  // M/N-contiguous operand: one box of 64 k rows x 64 elements
constexpr int SMEM_MAX = 232448;
constexpr int OUT_BOX_BYTES = 32 * 128;   // contract: 32 rows x 64 columns, staged for a TMA store
constexpr int OUT_BYTES = EPI_WARPS * 2 * OUT_BOX_BYTES;  // two boxes per epilogue warp
constexpr int CHUNK_COLS = 32;            // split: columns are exchanged in chunks of 32

// Division of 0 <= n < 2^31 by a number that is the same for a whole launch: every role of the kernel turns schedule positions
// into tiles, and two divisions by variables take it 500 cycles per tile.
struct Div {
  uint32_t mul, shift;  // mul 0: division by one
  __host__ static Div by(int d) {  // mul = ceil(2^(31 + l) / d), 2^(l - 1) < d <= 2^l: mul * d exceeds 2^(31 + l) by less than 2^l
    if (d <= 1) return {0u, 0u};
    uint32_t l = 1;
    while ((1ull << l) < static_cast<uint64_t>(d)) ++l;
    return {static_cast<uint32_t>(((1ull << (31 + l)) + d - 1) / d), l - 1};
  }
  __host__ __device__ int of(int n) const {
    if (mul == 0u) return n;
    return static_cast<int>(static_cast<uint32_t>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> 32) >> shift);
  }
};

enum Kind { DENSE = 0, ROWS = 1, CONTRACT = 2 };
// What the epilogue does besides the bias: nothing; the activation (runtime kind), with
// the value before it kept if asked for; the product with the activation's slope.
enum Epi { EPI_PLAIN = 0, EPI_ACT = 1, EPI_SLOPE = 2 };
enum Act { ACT_NONE = 0, ACT_GELU = 1, ACT_RELU = 2, ACT_SILU = 3 };

struct alignas(64) Params {
  CUtensorMap tmA, tmB;
  CUtensorMap tmOut;  // contract: the output, written with TMA stores
  int M, N, K;
  int MBQ, NB, KB;   // scheduling blocks (128 or 256 rows), column blocks, k blocks of the whole contraction
  int bn;            // tile columns
  int group;         // scheduling blocks swept together (rasterisation)
  Div per, first, last;  // dense: by group * NB, group and the size of the last group; rows: by NB; contract: by MBQ * NB and MBQ
  int groups;
  int split;         // members of a cluster that share a tile
  int stages, a_slot, b_slot;  // operand ring: bytes per stage
  int a_whole, b_whole;  // M/N-contiguous operand whose extent is a multiple of 64: one box of a 4-D map holds a stage's share
  int a_rows;        // rows of A a stage brings in (128 per half, or fewer when M or the groups are smaller)
  int slot_rows;     // split: rows of an exchange slot (128, or fewer when M is smaller)
  int wide;          // rows of the output start at multiples of 32 bytes: whole-sector stores
  int act;           // applied to the rounded result, or, with pre_in, its derivative at pre_in
  const bf16* bias;
  float bias_scale;
  const bf16* w;       // the weights where the first of them may be prefetched, or null
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

// exp(-|x|) cannot overflow, so the sigmoid of a negative number keeps its leading digits down to the smallest
// fp32 value (1 / (1 + exp(-x)) with the fast division is 0 from -87.3 on).  The fast exponential and division
// stay far inside the bf16 rounding that follows: over all finite bf16 inputs SiLU, GELU and their slopes round to the
// nearest bf16 value except for 3 of 261120 (torch's own, with expf, tanhf and full division: 347).  expf and full
// division here cost 10 us of a MoE layer's 104 (32 tokens) and 29 us of a training step's 519.
__device__ __forceinline__ float sigmoid(float x) {
  const float t = __expf(-fabsf(x));
  return __fdividef(x < 0.0f ? t : 1.0f, 1.0f + t);
}
// tanh form of GELU: x * sigmoid(2u), u = sqrt(2/pi) * (x + 0.044715 x^3)
constexpr float GELU_C = 2.0f * 0.7978845608028654f;
constexpr float GELU_A = 0.044715f;
template <int kAct>
__device__ __forceinline__ float act_value(float x) {
  if constexpr (kAct == ACT_GELU) return x * sigmoid(GELU_C * x * (1.0f + GELU_A * x * x));
  else if constexpr (kAct == ACT_SILU) return x * sigmoid(x);
  else return x < 0.0f ? 0.0f : x;
}
template <int kAct>
__device__ __forceinline__ float act_slope(float x) {
  if constexpr (kAct == ACT_GELU) {
    const float s = sigmoid(GELU_C * x * (1.0f + GELU_A * x * x));
    return s + x * s * (1.0f - s) * GELU_C * (1.0f + 3.0f * GELU_A * x * x);
  } else {
    const float s = sigmoid(x);
    return s * (1.0f + x * (1.0f - s));
  }
}
template <int kAct>
__device__ __forceinline__ void act32(const uint4* pre, uint4* out) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float s[8];
    unpack8(pre[i], s);
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = act_value<kAct>(s[e]);
    out[i] = pack8(s);
  }
}
template <int kAct>
__device__ __forceinline__ void slope32(const uint4* at, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float s[8];
    unpack8(at[i], s);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      // ReLU selects: an infinite gradient where it is off is zero, a NaN passes the gradient on
      if constexpr (kAct == ACT_RELU) f[8 * i + e] = s[e] <= 0.0f ? 0.0f : f[8 * i + e];
      else f[8 * i + e] *= act_slope<kAct>(s[e]);
    }
  }
}

// 32 accumulator values of one row -> bf16: (+ bias, one rounding), then the activation
// of the rounded value, or the product with the slope at the saved value `at`.  A scheduler has two
// epilogue warps at most, so latency counts: all loads of the 32 columns are issued
// together and the arithmetic is straight-line, branches are taken once per 32 columns
// (branching per 8 values cost 250 cycles each: 11000 cycles for a 128 x 256 tile).
template <Epi kEpi>
__device__ __forceinline__ void finish32(const Params& p, float* f, int col, const uint4* at, uint4* out, uint4* pre) {
  if (p.bias != nullptr) {
    uint4 b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = col + 8 * i < p.N ? kb::ld_global_v4(p.bias + col + 8 * i) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float t[8];
      unpack8(b[i], t);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[8 * i + e] += p.bias_scale * t[e];
    }
  }
  if constexpr (kEpi == EPI_SLOPE) {
    if (p.act == ACT_SILU) slope32<ACT_SILU>(at, f);
    else if (p.act == ACT_GELU) slope32<ACT_GELU>(at, f);
    else slope32<ACT_RELU>(at, f);
  }
  uint4* rounded = kEpi == EPI_ACT ? pre : out;
#pragma unroll
  for (int i = 0; i < 4; ++i) rounded[i] = pack8(f + 8 * i);
  if constexpr (kEpi == EPI_ACT) {
    if (p.act == ACT_SILU) act32<ACT_SILU>(pre, out);
    else if (p.act == ACT_GELU) act32<ACT_GELU>(pre, out);
    else act32<ACT_RELU>(pre, out);
  }
}
// 32 values of a lane's row, straight from the registers.  A lane's 32-byte store is a
// whole L2 sector, so the 32 rows a warp touches per instruction cost no partial
// writes.  Staging through shared memory (for TMA stores, or to let eight lanes store
// a row's 128 bytes) moves twice the tile through a memory whose bandwidth a pair's
// mainloop uses up: operands in and out are 128 bytes per cycle.  It also costs a
// pipeline stage; 8 groups of 1000 rows, 4096 x 4096: 198 us stored from registers, 207 staged.
__device__ __forceinline__ void store_row32(bf16* base, size_t at, int col, int n, bool wide, const uint4* v) {
  if (wide && col + 32 <= n) {
    kb::st_global_v8(base + at, v[0], v[1]);
    kb::st_global_v8(base + at + 16, v[2], v[3]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (col + 8 * i < n) *reinterpret_cast<uint4*>(base + at + 8 * i) = v[i];
  }
}

// Saved values of 32 columns from `c` on of a tile's row; `last`: columns that exist.
__device__ __forceinline__ void fetch32(const Params& p, const bf16* row, int c, int last, uint4* at) {
  if (p.wide && c + 32 <= last) {
    kb::ld_stream_v8(row + c, at[0], at[1]);
    kb::ld_stream_v8(row + c + 16, at[2], at[3]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    at[i] = make_uint4(0u, 0u, 0u, 0u);
    if (c + 8 * i < last) at[i] = kb::ld_stream_v4(row + c + 8 * i);
  }
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

// Weights on their way into the L2 before the previous launch has ended: the first k blocks of `cols` columns from `col` on,
// by 256 threads.  Nothing is read by it, so it does not matter that someone may still write them.  `w`: [N][K].
constexpr int AHEAD = 12;  // k blocks, 30 MB on 148 SMs: with 6 half of the gain, with 20 and 32 no more
__device__ __forceinline__ void prefetch_weights(const bf16* w, int N, int K, int col, int cols, int k0, int k1, int thread) {
  const int k = k0 * BK, ks = min(min(k1 - k0, AHEAD) * BK, K - k);
  const int cs = min(cols, N - col);
  if (ks <= 0) return;
  for (int i = thread; i < cs; i += 256) kb::prefetch_l2(w + static_cast<size_t>(col + i) * K + k, static_cast<uint32_t>(ks) * 2);
}

// kHalves: 128-row blocks per CTA and tile.  2 (pairs only): a 512-row tile whose two
// halves fill both accumulators.
template <Kind kKind, bool kPair, bool kAMn, bool kBMn, int kHalves, Epi kEpi>
__global__ void __launch_bounds__(THREADS, 1) gemm_local_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sm_a = base;
  uint8_t* sm_b = sm_a + p.stages * p.a_slot;
  uint8_t* sm_out = sm_b + p.stages * p.b_slot;  // 1024-byte aligned: slots are multiples of eight 128-byte rows
  uint8_t* sm_bar = sm_out + (kKind == CONTRACT ? OUT_BYTES : 0);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm_bar);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= BAR_BYTES, "barrier block too small");
  int32_t* pref = reinterpret_cast<int32_t*>(sm_bar + BAR_BYTES);  // [groups + 1] row blocks before a group
  int32_t* g_start = pref + p.groups + 1;                                      // [groups]
  int32_t* g_count = g_start + p.groups;                                       // [groups]

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
      const int g = p.per.of(pos);
      const int r = pos - g * p.group * p.NB;
      const int gs = min(p.MBQ - g * p.group, p.group);
      nb = (gs == p.group ? p.first : p.last).of(r);
      mbq = g * p.group + (r - nb * gs);
      t.group = 0;
      t.row0 = mbq * TILE_ROWS + static_cast<int>(half) * CTA_ROWS;
      t.row_end = p.M;
    } else if constexpr (kKind == ROWS) {
      const int block = p.per.of(pos);  // counts row blocks: group e holds blocks pref[e] .. pref[e + 1] - 1
      int lo = 0, hi = p.groups - 1;
      while (lo < hi) {  // last group with pref <= block: it is not empty
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= block) lo = mid;
        else hi = mid - 1;
      }
      const int blocks = pref[lo + 1] - pref[lo];
      const int r = pos - pref[lo] * p.NB;
      nb = blocks == 1 ? r : r / blocks;
      mbq = r - nb * blocks;
      t.group = lo;
      t.row0 = g_start[lo] + mbq * block_rows + static_cast<int>(half) * CTA_ROWS;
      t.row_end = min(g_start[lo] + g_count[lo], t.row0 + (kPair ? CTA_ROWS : block_rows));
    } else {
      t.group = p.per.of(pos);
      const int r = pos - t.group * p.MBQ * p.NB;
      nb = p.first.of(r);
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
  // (at most 2^25 of them and eight members: 32 bits hold the products)
  auto k_range = [&](const Tile& t, int& k0, int& k1) {
    k0 = 0;
    k1 = t.kb;
    if (kKind == DENSE && p.split > 1) {
      k0 = static_cast<int>(static_cast<uint32_t>(t.kb * member) / static_cast<uint32_t>(p.split));
      k1 = static_cast<int>(static_cast<uint32_t>(t.kb * (member + 1)) / static_cast<uint32_t>(p.split));
    }
  };

  if (warp == 0) {
    if (lane < p.stages) {
      kb::mbar_init(&full[lane], 1);
      kb::mbar_init(&empty[lane], 1);
    }
    if (lane < 2) {
      kb::mbar_init(&tfull[lane], 1);
      kb::mbar_init(&tempty[lane], kPair ? 2 * EPI_WARPS : EPI_WARPS);
    }
    if (lane == 0) *abort_flag = 0;
    kb::mbar_fence_init();
    __syncwarp();
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
  }
  if (kKind == DENSE && !kBMn && warp >= 4 && p.w != nullptr) {
    const Tile t = tile_at(sched_id);
    int k0, k1;
    k_range(t, k0, k1);
    prefetch_weights(p.w, p.N, p.K, t.n0 + static_cast<int>(half) * b_cols, b_cols, k0, k1, tid - 128);
  }
  kb::wait_for_previous_launch();  // barriers, tensor memory and descriptors are set up under the end of that one
  const uint64_t t_start = p.timing ? kb::globaltimer_ns() : 0;  // the product's own time
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
  // A pair's CTAs signal each other's barriers: both must have initialised theirs.
  // Otherwise the producer warp, which needs only the barriers it has just made,
  // goes ahead: its first loads are under way while the tensor memory is allocated.
  if constexpr (kPair) {
    kb::tc_fence_before_sync();
    __syncthreads();
    kb::cluster_sync_all();
    kb::tc_fence_after_sync();
  } else if (kKind == DENSE && warp == 0) {
    asm volatile("bar.arrive 1, %0;" ::"n"(THREADS) : "memory");
  } else {
    kb::tc_fence_before_sync();
    if constexpr (kKind == DENSE) asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    else __syncthreads();
    kb::tc_fence_after_sync();
  }
  const uint32_t tmem_base = (kPair || kKind != DENSE || warp != 0) ? *tmem_slot : 0u;

  const int total_tiles = kKind == DENSE ? p.MBQ * p.NB : kKind == ROWS ? pref[p.groups] * p.NB : p.groups * p.MBQ * p.NB;

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer ----
    // Converged like the MMA issuer: with few rows a stage is small and has to leave
    // every 350 cycles to keep the memory busy.
    {
      uint32_t s = 0;
      uint32_t ph = 0;
      bool ok = true;
      const uint32_t a_bytes = static_cast<uint32_t>(p.a_rows) * BK * 2;
      const uint32_t stage_bytes = a_bytes + static_cast<uint32_t>(b_cols) * BK * 2;
      const uint32_t a0 = kb::smem_u32(sm_a), b0 = kb::smem_u32(sm_b), full0 = kb::smem_u32(full);
      // a pair's bytes are counted on the leader's barrier, which expects the sum
      const uint32_t tx_bytes = kPair ? 2 * stage_bytes : stage_bytes;
      const uint32_t bar0 = kPair ? kb::map_to_cta(full0, lead) : full0;
      // M/N-contiguous operands in one load each instead of one per 64 columns where their extent allows it: issuing six loads per
      // stage is what held the producer back where a tile has few k blocks (weight gradients of 64 experts of 2048 x 1024, 128 rows:
      // 73.8 -> 70.8 us, on 32 SMs alone 276 -> 237).  Each kind of load has a loop of its own: with the choice inside it the loads per
      // 64 columns took a pair 3 to 8 % longer (16 groups of 808 rows, 1296 x 2400: 105.7 us, 98.9 here).
      auto produce = [&](auto a_whole, auto b_whole) {
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
            const uint32_t da = a0 + s * p.a_slot, db = b0 + s * p.b_slot, bar = bar0 + 8 * s, own = full0 + 8 * s;
            if (++s == static_cast<uint32_t>(p.stages)) {
              s = 0;
              ph ^= 1u;
            }
            if constexpr (!kAMn && !kBMn) {
              kb::tma_load_ab_warp<kPair>(own, leader ? tx_bytes : 0u, bar, da, &p.tmA, k * BK, t.row0, 0, db, &p.tmB, k * BK, nrow, bz);
              continue;
            }
            if (leader) kb::mbar_expect_tx_warp(own, tx_bytes);
            if constexpr (!kAMn) {
              kb::tma_load_3d_warp<kPair>(da, &p.tmA, bar, k * BK, t.row0, 0);
            } else if constexpr (decltype(a_whole)::value) {
              kb::tma_load_4d_warp<kPair>(da, &p.tmA, bar, 0, t.k_row + k * BK, t.row0 / 64, 0);
            } else {
#pragma unroll
              for (int i = 0; i < CTA_ROWS / 64; ++i) {
                kb::tma_load_3d_warp<kPair>(da + i * MN_BLOCK_BYTES, &p.tmA, bar, t.row0 + i * 64, t.k_row + k * BK, 0);
              }
            }
            if constexpr (!kBMn) {
              kb::tma_load_3d_warp<kPair>(db, &p.tmB, bar, k * BK, nrow, bz);
            } else if constexpr (decltype(b_whole)::value) {
              kb::tma_load_4d_warp<kPair>(db, &p.tmB, bar, 0, t.k_row + k * BK, nrow / 64, bz);
            } else {
              for (int i = 0; i < b_cols / 64; ++i) {
                kb::tma_load_3d_warp<kPair>(db + i * MN_BLOCK_BYTES, &p.tmB, bar, nrow + i * 64, t.k_row + k * BK, bz);
              }
            }
          }
        }
      };
      using Yes = std::true_type;
      using No = std::false_type;
      if constexpr (kAMn) {
        if (p.a_whole && p.b_whole) produce(Yes{}, Yes{});
        else if (p.a_whole) produce(Yes{}, No{});
        else if (p.b_whole) produce(No{}, Yes{});
        else produce(No{}, No{});
      } else if constexpr (kBMn) {
        if (p.b_whole) produce(No{}, Yes{});
        else produce(No{}, No{});
      } else {
        produce(No{}, No{});
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
      // A k block of a narrow tile takes the tensor pipe 256 cycles: nothing that is the same
      // for all k blocks of a tile is decided inside the loop over them (which halves take
      // part, first use of the accumulator, empty groups: 464 -> 300 cycles per block).
      for (int pos = sched_id; pos < total_tiles; pos += sched_n, ++it) {
        const Tile t = tile_at(pos);
        int k0, k1;
        k_range(t, k0, k1);
        // one half: accumulators alternate from tile to tile; two halves: a tile fills both
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {
          const uint32_t acc = kHalves == 2 ? static_cast<uint32_t>(h) : it & 1u;
          const uint32_t use = kHalves == 2 ? it : it >> 1;
          if (ok && !kb::mbar_wait_bounded(&tempty[acc], (use & 1u) ^ 1u, p.limit_ns)) {
            kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_TEMPTY, (uint32_t)pos, 0);
            ok = false;
          }
        }
        if (!ok) break;
        kb::tc_fence_after_sync();
        const uint32_t d = tmem_base + (kHalves == 2 ? 0u : (it & 1u) * ACC_COLS);
        uint32_t accumulate = 0;
        for (int left = k1 - k0; left > 0; --left) {
          if (!kb::mbar_wait_bounded(&full[s], ph, p.limit_ns)) {
            kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, SITE_FULL, (uint32_t)pos, 0);
            ok = false;
            break;
          }
          kb::tc_fence_after_sync();
          const uint32_t sa = a_lo + s * a_inc, sb = b_lo + s * b_inc, bar = s * 8;
          if (++s == static_cast<uint32_t>(p.stages)) {
            s = 0;
            ph ^= 1u;
          }
#pragma unroll
          for (int h = 0; h < kHalves; ++h) {
            kb::umma_f16_x4<kPair>(d + h * ACC_COLS, sa + h * (BM * BK * 2 / 16), a_hi, sb, b_hi, A_STEP, B_STEP, idesc, accumulate);
          }
          accumulate = 1;
          // the stage is free (in both CTAs of a pair) once these MMAs have read it
          kb::umma_commit_warp<kPair>(empty0 + bar);
          if constexpr (kPair) kb::umma_commit_warp<kPair>(empty1 + bar);
        }
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < kHalves; ++h) {  // an empty group hands its accumulator on as well
          const uint32_t f = kb::smem_u32(&tfull[kHalves == 2 ? static_cast<uint32_t>(h) : it & 1u]);
          kb::umma_commit_warp<kPair>(kPair ? kb::map_to_cta(f, lead) : f);
          if constexpr (kPair) kb::umma_commit_warp<kPair>(kb::map_to_cta(f, lead + 1u));
        }
      }
      if (!ok) *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp >= 4 && p.split == 1) {
    // ---------------------------------------------------------- epilogue ----
    // Warps q and q + 4 of the role drain lane quadrant q, 64 columns in turn.
    const int q = warp & 3;
    const int turn = (warp - 4) >> 2;
    uint32_t it = 0;
    int box_no = 0;  // contract: staging boxes used by this warp
    for (int pos = sched_id; pos < total_tiles; pos += sched_n, ++it) {
      const Tile t = tile_at(pos);
      if constexpr (kEpi == EPI_SLOPE) {
        // The tile's saved values are on their way from memory while its products are made: a lane's row of it, 64 columns in turn
        // as below.
        for (int hb = 0; hb < kHalves; ++hb) {
          const int row = t.row0 + hb * BM + q * 32 + lane;
          for (int c = turn * 64; c < p.bn && row < t.row_end && t.n0 + c < p.N; c += 128) {
            kb::prefetch_l2(p.pre_in + static_cast<size_t>(row) * p.N + t.n0 + c, min(64, p.N - t.n0 - c) * 2);
          }
        }
      }
      if (p.bias != nullptr) {
        // brings the tile's bias into L1 while the accumulator is not ready yet: eight values per lane
        const int col = t.n0 + 8 * lane;
        if (8 * lane < p.bn && col < p.N) kb::touch_global(p.bias + col);
      }
      const int cols = min(p.bn, p.N - t.n0);
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
        auto release = [&]() {  // this warp has read its share of the accumulator
          kb::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) {
              if (leader) kb::mbar_arrive(&tempty[acc]);
              else kb::mbar_arrive_cluster_relaxed(kb::map_to_cta(kb::smem_u32(&tempty[acc]), lead));
            } else {
              kb::mbar_arrive(&tempty[acc]);
            }
          }
        };
        const int last = gr0 < t.row_end ? cols : 0;
        if (turn * 64 >= last) release();
        if constexpr (kEpi == EPI_SLOPE) {
          // 32 columns at a time, the saved values one step ahead.
          uint4 at[4], next[4];
          const bf16* saved = p.pre_in + static_cast<size_t>(row) * p.N + t.n0;
          const int mine = row_ok ? last : 0;
          fetch32(p, saved, turn * 64, mine, at);
#pragma unroll 1
          for (int s = 0; s < 4; ++s) {  // columns turn * 64 + 0, 32, 128, 160
            const int c = turn * 64 + (s >> 1) * 128 + (s & 1) * 32;
            if (c >= last) break;
            const int c1 = c + ((s & 1) ? 96 : 32);
            if (s < 3) fetch32(p, saved, c1, mine, next);
            uint32_t r[32];
            kb::tmem_ld_32x32(taddr + c, r);
            kb::tmem_ld_wait();
            if (s == 3 || c1 >= last) release();
            float f[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
            uint4 o[4], pre[4];
            finish32<kEpi>(p, f, t.n0 + c, at, o, pre);
            if (row_ok) store_row32(p.out, static_cast<size_t>(row) * p.N + t.n0 + c, t.n0 + c, p.N, p.wide != 0, o);
#pragma unroll
            for (int i = 0; i < 4; ++i) at[i] = next[i];
          }
          continue;
        }
        if constexpr (kKind == CONTRACT) {
          // Few k blocks per tile: the output is the traffic.  Staged boxes leave as whole
          // 128-byte lines while the epilogue goes on (rows and columns outside the tensor are
          // clipped); unlike in a long contraction the mainloop leaves shared memory
          // bandwidth for it.  64 experts, 128 rows, 2048 x 1024: 85 us stored from registers,
          // 75 staged; writing 268 MB alone takes a memset 72.
#pragma unroll 1
          for (int c = turn * 64; c < last; c += 128) {
            uint8_t* box = sm_out + ((warp - 4) * 2 + (box_no++ & 1)) * OUT_BOX_BYTES;
            uint32_t r[2][32];
            if (t.kb == 0) {  // an empty group: nothing was accumulated
#pragma unroll
              for (int i = 0; i < 32; ++i) r[0][i] = r[1][i] = 0u;
            } else {
              kb::tmem_ld_32x32(taddr + c, r[0]);
              kb::tmem_ld_32x32(taddr + c + 32, r[1]);
            }
            if (lane == 0) kb::bulk_wait_group_read<1>();  // the box's previous store has read it
            __syncwarp();
            if (t.kb != 0) kb::tmem_ld_wait();
            if (c + 128 >= last) release();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[j >> 2][(j & 3) * 8 + e]);
              *reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) * 16)) = pack8(f);
            }
            kb::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              kb::tma_store_3d(&p.tmOut, box, t.n0 + c, gr0, t.group);
              kb::bulk_commit_group();
            }
          }
          continue;
        }
#pragma unroll 1
        for (int c = turn * 64; c < last; c += 128) {
          const bool two = c + 32 < last;
          const int col = t.n0 + c;
          const size_t at0 = static_cast<size_t>(row) * p.N + col;
          uint32_t r[2][32];
          kb::tmem_ld_32x32(taddr + c, r[0]);
          if (two) kb::tmem_ld_32x32(taddr + c + 32, r[1]);
          kb::tmem_ld_wait();
          if (c + 128 >= last) release();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && !two) break;
            float f[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[h][i]);
            uint4 o[4], pre[4];
            finish32<kEpi>(p, f, col + 32 * h, nullptr, o, pre);
            if (row_ok) {
              store_row32(p.out, at0 + 32 * h, col + 32 * h, p.N, p.wide != 0, o);
              if constexpr (kEpi == EPI_ACT) {
                if (p.pre_out != nullptr) store_row32(p.pre_out, at0 + 32 * h, col + 32 * h, p.N, p.wide != 0, pre);
              }
            }
          }
        }
      }
    }
    if (kKind == CONTRACT && lane == 0) kb::bulk_wait_group<0>();
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
      // source) of the owner's operand ring holds slot_rows x 32 columns as
      // [4-column group][row] float4: neighbouring lanes write neighbouring 16 bytes.
      __syncthreads();
      kb::cluster_sync_all();  // every member's MMAs have finished: all operand rings are free
      kb::tc_fence_after_sync();
      const uint32_t tmem_base = *tmem_slot;  // the producer warp did not wait for it
      const Tile t = tile_at(sched_id);
      if (p.bias != nullptr) {
        const int col = t.n0 + 8 * lane;
        if (8 * lane < p.bn && col < p.N) kb::touch_global(p.bias + col);
      }
      const int chunks = p.bn / CHUNK_COLS;
      const int q = warp & 3;            // TMEM lane quadrant of this warp
      const int gr0 = t.row0 + q * 32;
      const int row = gr0 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      const int slot_bytes = p.slot_rows * CHUNK_COLS * 4;
      const bool live = gr0 < t.row_end;
      if (live) {
        for (int c = warp >> 2; c < chunks; c += THREADS / 128) {
          const int owner = c * p.split / chunks;
          if (owner == member || t.n0 + c * CHUNK_COLS >= p.N) continue;
          const int first = (owner * chunks + p.split - 1) / p.split;  // the owner's first chunk
          const int src = member < owner ? member : member - 1;
          uint32_t r[32];
          kb::tmem_ld_32x32(taddr + c * CHUNK_COLS, r);
          kb::tmem_ld_wait();
          const uint32_t to = kb::map_to_cta(kb::smem_u32(base + ((c - first) * (p.split - 1) + src) * slot_bytes),
                                             static_cast<uint32_t>(owner) * (kPair ? 2u : 1u) + half);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            kb::st_shared_cluster_v4(to + (i * p.slot_rows + q * 32 + lane) * 16, r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
          }
        }
      }
      kb::cluster_sync_all();  // the partials are in place
      if (live) {
        for (int c = warp >> 2; c < chunks; c += THREADS / 128) {
          const int col0 = t.n0 + c * CHUNK_COLS;
          if (c * p.split / chunks != member || col0 >= p.N) continue;
          const int first = (member * chunks + p.split - 1) / p.split;
          uint32_t r[32];
          kb::tmem_ld_32x32(taddr + c * CHUNK_COLS, r);
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = 0.f;
          const uint32_t from = kb::smem_u32(base) + (q * 32 + lane) * 16;
          kb::tmem_ld_wait();
#pragma unroll 1
          for (int m = 0; m < p.split; ++m) {  // ascending member order
            if (m == member) {
#pragma unroll
              for (int i = 0; i < 32; ++i) f[i] += __uint_as_float(r[i]);
            } else {
              const uint32_t slot = from + ((c - first) * (p.split - 1) + (m < member ? m : m - 1)) * slot_bytes;
              float4 v[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = kb::ld_shared_v4(slot + i * p.slot_rows * 16);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                f[4 * i] += v[i].x; f[4 * i + 1] += v[i].y; f[4 * i + 2] += v[i].z; f[4 * i + 3] += v[i].w;
              }
            }
          }
          uint4 o[4], pre[4];
          uint4 at4[4];
          if constexpr (kEpi == EPI_SLOPE) {
            const uint4* src = reinterpret_cast<const uint4*>(p.pre_in + static_cast<size_t>(row) * p.N + col0);
#pragma unroll
            for (int i = 0; i < 4; ++i) at4[i] = row < t.row_end && col0 + 8 * i < p.N ? src[i] : make_uint4(0u, 0u, 0u, 0u);
          }
          finish32<kEpi>(p, f, col0, at4, o, pre);
          if (row < t.row_end) {
            const size_t at = static_cast<size_t>(row) * p.N + col0;
            store_row32(p.out, at, col0, p.N, p.wide != 0, o);
            if constexpr (kEpi == EPI_ACT) {
              if (p.pre_out != nullptr) store_row32(p.pre_out, at, col0, p.N, p.wide != 0, pre);
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
