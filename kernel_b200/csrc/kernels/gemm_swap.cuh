// Products with exchanged operands (host side: gemm_swap.cu): the weights are the MMA's M side, the token rows its N side.
//
//   dense     out[M,N] = X[M,K] * W[N,K]^T  with few rows M
//   rows      rows of X are grouped (one group per expert); group e is multiplied by its own W[e]
//
// The M side of tcgen05.mma comes in 128 (one CTA) or 256 (CTA pair) lanes, the N side in multiples of 16 (32 for a pair).
// With token rows on the M side a batch of 3 or of 137 rows pays for 128 or 256; here it pays for 16 or 144 (160), in
// tensor time, in shared memory traffic and, what counts most under the power cap, in energy.  64 experts of
// 2048 x 1024 and back, 32 tokens, top-6: a layer 108 -> 95 us.
//
// Warps 0 and 3 are the TMA producers of weights and tokens, warp 1 the MMA issuer, warp 2 owns the TMEM allocation,
// warps 4 to 11 are the epilogue.  Two accumulators of up to 256 token columns.  An accumulator lane is an output column, so a
// lane's values of neighbouring tokens are exchanged with three other lanes by shuffles until it holds four
// neighbouring columns of a token: 8-byte accesses that fill whole sectors.
//
// `early`: what the weights and the row table hold was written before the previous launch of the stream began (the
// caller's promise), so the first weight tiles are fetched under that launch's end; the token rows are not.  (16 x
// 7168 x 18432 back to back: 45.8 us, 44.0 with it.)
//
// Split contraction (dense): as in gemm_local.cuh, but the fp32 partial tiles are dealt out by token columns.
#pragma once
#include "gemm_local.cuh"

namespace kbs {

using kbl::bf16;
using kbl::Epi;
using kbl::EPI_ACT;
using kbl::EPI_PLAIN;
using kbl::EPI_SLOPE;
using kbl::Kind;
using kbl::DENSE;
using kbl::ROWS;

constexpr int BK = 64;
constexpr int LANES = 128;  // output columns of a CTA
constexpr int ACC_COLS = 256;
constexpr int TMEM_COLS = 512;
constexpr int THREADS = 384;
constexpr int EPI_WARPS = 8;
constexpr int MAX_STAGES = 16;
constexpr int BAR_BYTES = 512;
constexpr int CHUNK = 8;  // token columns of an exchange unit

struct alignas(64) Params {
  CUtensorMap tmW, tmX;
  int M, N, K;
  int NB, KB, MB;      // column blocks, k blocks, token blocks (dense)
  kbl::Div per;        // by MB (dense) or NB (rows)
  int bn;              // columns of a tile (both CTAs of a pair)
  int tok;             // most tokens of a tile, a multiple of 16 (one CTA) or 32 (pair)
  int xbox;            // rows of one box of X
  int groups, split;
  int stages, w_slot, x_slot;
  int w_whole;         // weights contiguous along N, a multiple of 64 of them: one box of a 4-D map holds a stage's columns
  int act;
  int early;
  const bf16* bias;
  float bias_scale;
  const bf16* w;       // the weights where the first of them may be prefetched, or null
  bf16* out;
  bf16* pre_out;
  const bf16* pre_in;
  const int32_t* row_start;
  const int32_t* row_count;
  uint32_t* status;
  uint64_t limit_ns;
  int timing;
};

struct Tile {
  int group;
  int row0, rows;  // first token row, tokens
  int cols;        // MMA columns: tokens rounded up to 16 (one CTA) or 32 (pair)
  int n0;          // first output column of the tile
};

// 2 * NV tokens of one column, packed in pairs, <-> NV / 2 groups of four neighbouring columns of one token: vector j of a lane
// is token 4 j + (lane & 3), columns (lane & ~3) .. + 3.
template <int NV>
__device__ __forceinline__ void to_rows(const uint32_t* v, uint2* o, int lane) {
  const bool odd = lane & 1, high = lane & 2;
  uint32_t u[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, v[i], 1);
    u[i] = odd ? __byte_perm(other, v[i], 0x7632) : __byte_perm(v[i], other, 0x5410);
  }
#pragma unroll
  for (int j = 0; j < NV / 2; ++j) {
    const uint32_t keep = high ? u[2 * j + 1] : u[2 * j];
    const uint32_t recv = __shfl_xor_sync(0xffffffffu, high ? u[2 * j] : u[2 * j + 1], 2);
    o[j] = high ? make_uint2(recv, keep) : make_uint2(keep, recv);
  }
}
template <int NV>
__device__ __forceinline__ void to_cols(const uint2* o, uint32_t* v, int lane) {
  const bool odd = lane & 1, high = lane & 2;
  uint32_t u[NV];
#pragma unroll
  for (int j = 0; j < NV / 2; ++j) {
    const uint32_t recv = __shfl_xor_sync(0xffffffffu, high ? o[j].x : o[j].y, 2);
    u[2 * j] = high ? recv : o[j].x;
    u[2 * j + 1] = high ? o[j].y : recv;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, u[i], 1);
    v[i] = odd ? __byte_perm(other, u[i], 0x7632) : __byte_perm(u[i], other, 0x5410);
  }
}
template <int kAct>
__device__ __forceinline__ uint32_t act2(uint32_t v) {
  const float2 f = kb::unpack_bf16x2(v);
  return kb::pack_bf16x2(kbl::act_value<kAct>(f.x), kbl::act_value<kAct>(f.y));
}
template <int kAct, int NV>
__device__ __forceinline__ void act_rows(const uint2* pre, uint2* o) {
#pragma unroll
  for (int j = 0; j < NV / 2; ++j) o[j] = make_uint2(act2<kAct>(pre[j].x), act2<kAct>(pre[j].y));
}
template <int kAct, int NV>
__device__ __forceinline__ void slope_cols(const uint32_t* at, float* f) {
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float2 s = kb::unpack_bf16x2(at[i]);
    if constexpr (kAct == kbl::ACT_RELU) {
      f[2 * i] = s.x <= 0.0f ? 0.0f : f[2 * i];
      f[2 * i + 1] = s.y <= 0.0f ? 0.0f : f[2 * i + 1];
    } else {
      f[2 * i] *= kbl::act_slope<kAct>(s.x);
      f[2 * i + 1] *= kbl::act_slope<kAct>(s.y);
    }
  }
}

// Row vectors of the saved values (EPI_SLOPE), fetched before the accumulator is read.
template <int NV>
__device__ __forceinline__ void fetch_saved(const Params& p, size_t at, int tokens, bool col_ok, int lane, uint2* saved) {
#pragma unroll
  for (int j = 0; j < NV / 2; ++j) {
    const int t = 4 * j + (lane & 3);
    saved[j] = make_uint2(0u, 0u);
    if (col_ok && t < tokens) saved[j] = kb::ld_stream_v2(p.pre_in + at + static_cast<size_t>(t) * p.N);
  }
}
// 2 * NV fp32 results of one output column -> bf16 rows: bias, slope, one rounding, activation of the rounded value.  `at`: offset
// of the first token's vector; `tokens`: how many of them exist.
template <Epi kEpi, int NV>
__device__ __forceinline__ void finish(const Params& p, float* f, float bias, const uint2* saved, size_t at, int tokens, bool col_ok, int lane) {
  if (p.bias != nullptr) {
#pragma unroll
    for (int i = 0; i < 2 * NV; ++i) f[i] += bias;
  }
  if constexpr (kEpi == EPI_SLOPE) {
    uint32_t s[NV];
    to_cols<NV>(saved, s, lane);
    if (p.act == kbl::ACT_SILU) slope_cols<kbl::ACT_SILU, NV>(s, f);
    else if (p.act == kbl::ACT_GELU) slope_cols<kbl::ACT_GELU, NV>(s, f);
    else slope_cols<kbl::ACT_RELU, NV>(s, f);
  }
  uint32_t v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = kb::pack_bf16x2(f[2 * i], f[2 * i + 1]);
  uint2 rows[NV / 2], value[NV / 2];
  to_rows<NV>(v, rows, lane);
  if constexpr (kEpi == EPI_ACT) {
    if (p.act == kbl::ACT_SILU) act_rows<kbl::ACT_SILU, NV>(rows, value);
    else if (p.act == kbl::ACT_GELU) act_rows<kbl::ACT_GELU, NV>(rows, value);
    else act_rows<kbl::ACT_RELU, NV>(rows, value);
  }
  if (!col_ok) return;
#pragma unroll
  for (int j = 0; j < NV / 2; ++j) {
    const int t = 4 * j + (lane & 3);
    if (t >= tokens) continue;
    const size_t to = at + static_cast<size_t>(t) * p.N;
    *reinterpret_cast<uint2*>(p.out + to) = kEpi == EPI_ACT ? value[j] : rows[j];
    if constexpr (kEpi == EPI_ACT) {
      if (p.pre_out != nullptr) *reinterpret_cast<uint2*>(p.pre_out + to) = rows[j];
    }
  }
}

template <Kind kKind, bool kPair, bool kWMn, Epi kEpi>
__global__ void __launch_bounds__(THREADS, 1) gemm_swap_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sm_w = base;
  uint8_t* sm_x = sm_w + p.stages * p.w_slot;
  uint8_t* sm_bar = sm_x + p.stages * p.x_slot;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm_bar);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* tfull = empty + MAX_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  static_assert((2 * MAX_STAGES + 4) * 8 + 8 <= BAR_BYTES, "barrier block too small");
  int32_t* pref = reinterpret_cast<int32_t*>(sm_bar + BAR_BYTES);  // [groups + 1] token blocks before a group
  int32_t* g_start = pref + p.groups + 1;
  int32_t* g_count = g_start + p.groups;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const uint32_t ctarank = (kPair || p.split > 1) ? kb::cluster_ctarank() : 0u;
  const uint32_t half = kPair ? (ctarank & 1u) : 0u;        // which 128 output columns, and which half of the tokens it stages
  const uint32_t lead = kPair ? (ctarank & ~1u) : ctarank;  // cluster rank of the CTA that issues the MMAs
  const bool leader = half == 0u;
  const int member = static_cast<int>(kPair ? (ctarank >> 1) : ctarank);
  const int cta_per_tile = (kPair ? 2 : 1) * p.split;
  const int sched_id = static_cast<int>(blockIdx.x) / cta_per_tile;
  const int sched_n = static_cast<int>(gridDim.x) / cta_per_tile;
  constexpr int STEP = kPair ? 32 : 16;        // MMA columns come in multiples of this
  const int w_cols = kPair ? p.bn / 2 : p.bn;  // output columns of this CTA

  int k0 = 0, k1 = p.KB;  // this member's part (32 bits: at most 2^25 k blocks, eight members)
  if (kKind == DENSE && p.split > 1) {
    k0 = static_cast<int>(static_cast<uint32_t>(p.KB * member) / static_cast<uint32_t>(p.split));
    k1 = static_cast<int>(static_cast<uint32_t>(p.KB * (member + 1)) / static_cast<uint32_t>(p.split));
  }
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
    kb::tma_prefetch_desc(&p.tmW);
    kb::tma_prefetch_desc(&p.tmX);
  }
  if (kKind == DENSE && !kWMn && warp >= 4 && p.w != nullptr) {
    kbl::prefetch_weights(p.w, p.N, p.K, p.per.of(sched_id) * p.bn + static_cast<int>(half) * w_cols, w_cols, k0, k1, tid - 128);
  }
  if (!p.early) kb::wait_for_previous_launch();
  uint64_t t_start = p.timing ? kb::globaltimer_ns() : 0;  // the product's own time
  if constexpr (kKind == ROWS) {
    for (int e = tid; e < p.groups; e += THREADS) {
      g_start[e] = p.row_start[e];
      g_count[e] = p.row_count[e];
    }
    __syncthreads();
    if (warp == 0) {  // exclusive prefix of the groups' token blocks
      int carry = 0;
      for (int e0 = 0; e0 < p.groups; e0 += 32) {
        const int e = e0 + lane;
        int v = e < p.groups ? (g_count[e] + p.tok - 1) / p.tok : 0;
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
  // Both producers start from barriers that warp 0 has made; a pair's CTAs signal each other's.
  kb::tc_fence_before_sync();
  __syncthreads();
  if constexpr (kPair) kb::cluster_sync_all();
  kb::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = kKind == DENSE ? p.MB * p.NB : pref[p.groups] * p.NB;

  // Position in the static schedule -> tile.  The token blocks that share a panel of weights follow each other.
  auto tile_at = [&](int pos) -> Tile {
    Tile t;
    if constexpr (kKind == DENSE) {
      const int nb = p.per.of(pos);
      t.group = 0;
      t.row0 = (pos - nb * p.MB) * p.tok;
      t.rows = min(p.tok, p.M - t.row0);
      t.n0 = nb * p.bn;
    } else {
      const int block = p.per.of(pos);  // counts token blocks: group e holds blocks pref[e] .. pref[e + 1] - 1
      int lo = 0, hi = p.groups - 1;
      while (lo < hi) {  // last group with pref <= block: it is not empty
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= block) lo = mid;
        else hi = mid - 1;
      }
      const int blocks = pref[lo + 1] - pref[lo];
      const int r = pos - pref[lo] * p.NB;
      const int nb = blocks == 1 ? r : r / blocks, mb = r - nb * blocks;
      const int count = g_count[lo];
      const int most = blocks == 1 ? count : (count + blocks - 1) / blocks;
      const int per = (most + STEP - 1) / STEP * STEP;  // blocks of a group are alike; none is empty: per <= tok
      t.group = lo;
      t.row0 = g_start[lo] + mb * per;
      t.rows = min(per, count - mb * per);
      t.n0 = nb * p.bn;
    }
    t.cols = (t.rows + STEP - 1) / STEP * STEP;
    return t;
  };
  auto boxes_of = [&](const Tile& t) { return ((kPair ? t.cols >> 1 : t.cols) + p.xbox - 1) / p.xbox; };

  if (warp == 0) {
    // ------------------------------------------------ producer: weights ----
    // Two producers: with its barrier and coordinates a warp issues a load every 300 cycles at best, and narrow tiles need a
    // stage of weights that often (one producer: 320 ns per k block of 16 tokens and more with each box).  This one
    // announces the bytes of both.
    const uint32_t w0 = kb::smem_u32(sm_w), full0 = kb::smem_u32(full);
    const uint32_t bar0 = kPair ? kb::map_to_cta(full0, lead) : full0;
    const uint32_t w_bytes = static_cast<uint32_t>(w_cols) * BK * 2;
    const uint32_t box_bytes = static_cast<uint32_t>(p.xbox) * BK * 2;
    uint32_t s = 0, ph = 0;
    int ahead = p.early ? p.stages : -1;  // stages to fill before the previous launch has ended; then its end is no part of a bounded wait
    bool ok = true;
    for (int pos = sched_id; ok && pos < total_tiles; pos += sched_n) {
      const Tile t = tile_at(pos);
      const uint32_t bytes = (w_bytes + static_cast<uint32_t>(boxes_of(t)) * box_bytes) * (kPair ? 2 : 1);
      const int col = t.n0 + static_cast<int>(half) * w_cols;
      for (int k = k0; k < k1; ++k) {
        if (ahead >= 0 && ahead-- == 0) kb::wait_for_previous_launch();
        if (!kb::mbar_wait_bounded(&empty[s], ph ^ 1u, p.limit_ns, 400)) {
          kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_EMPTY, (uint32_t)pos, 0);
          *abort_flag = 1;
          ok = false;
          break;
        }
        const uint32_t own = full0 + 8 * s, bar = bar0 + 8 * s, dst = w0 + s * p.w_slot;
        if (++s == static_cast<uint32_t>(p.stages)) {
          s = 0;
          ph ^= 1u;
        }
        // A pair's bytes are counted on the leader's barrier.  Weights along N: one load instead of two per k block (input
        // gradients of 64 experts of 2048 x 1024, 3 rows each: 51.6 -> 44.8 us, 16 rows: 53.0 -> 50.1).
        if (kWMn && p.w_whole) {
          kb::tma_load_4d_expect_warp<kPair>(own, leader ? bytes : 0u, bar, dst, &p.tmW, 0, k * BK, col / 64, t.group);
          continue;
        }
        kb::tma_load_expect_warp<kPair>(own, leader ? bytes : 0u, bar, dst, &p.tmW, kWMn ? col : k * BK, kWMn ? k * BK : col, t.group);
        if constexpr (kWMn) {
          for (int i = 1; i < w_cols / 64; ++i) {
            kb::tma_load_3d_warp<kPair>(dst + i * kbl::MN_BLOCK_BYTES, &p.tmW, bar, col + i * 64, k * BK, t.group);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------- producer: tokens ----
    if (p.early) kb::wait_for_previous_launch();
    const uint32_t x0 = kb::smem_u32(sm_x), full0 = kb::smem_u32(full);
    const uint32_t bar0 = kPair ? kb::map_to_cta(full0, lead) : full0;
    const uint32_t box_bytes = static_cast<uint32_t>(p.xbox) * BK * 2;
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int pos = sched_id; ok && pos < total_tiles; pos += sched_n) {
      const Tile t = tile_at(pos);
      const int boxes = boxes_of(t);
      const int row = t.row0 + (kPair ? static_cast<int>(half) * (t.cols >> 1) : 0);
      for (int k = k0; k < k1; ++k) {
        if (!kb::mbar_wait_bounded(&empty[s], ph ^ 1u, p.limit_ns, 400)) {
          kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_EMPTY, (uint32_t)pos, 1);
          *abort_flag = 1;
          ok = false;
          break;
        }
        const uint32_t bar = bar0 + 8 * s, dst = x0 + s * p.x_slot;
        if (++s == static_cast<uint32_t>(p.stages)) {
          s = 0;
          ph ^= 1u;
        }
        // Boxes by twos: one by one this warp took 550 cycles per k block of two, the weights' 365 (input gradients of 64 experts of
        // 2048 x 1024, 128 rows each, on 74 SMs 95 -> 85 us).
        int i = 0;
        if constexpr (kKind == ROWS) {
          for (; i + 1 < boxes; i += 2) {
            kb::tma_load_3d_two_warp<kPair>(dst + i * box_bytes, dst + (i + 1) * box_bytes, &p.tmX, bar, k * BK, row + i * p.xbox, row + (i + 1) * p.xbox, 0);
          }
        }
        if (i < boxes) kb::tma_load_3d_warp<kPair>(dst + i * box_bytes, &p.tmX, bar, k * BK, row + i * p.xbox, 0);
      }
    }
    __syncwarp();
  } else {
    if (p.early) {
      kb::wait_for_previous_launch();
      if (p.timing) t_start = kb::globaltimer_ns();
    }
    if (warp == 1) {
      // ------------------------------------------------------ MMA issuer ----
      if (leader) {
        const uint32_t idesc0 = kb::umma_idesc_bf16(kPair ? 256 : 128, 0) | (kWMn ? 1u << 15 : 0u);
        constexpr uint32_t W_STEP = (kWMn ? kbl::UMMA_K * 128 : kbl::UMMA_K * 2) >> 4;
        constexpr uint32_t X_STEP = (kbl::UMMA_K * 2) >> 4;
        const uint64_t dw = kWMn ? kbl::desc_mn_sw128(kb::smem_u32(sm_w)) : kb::umma_desc_k_sw128(kb::smem_u32(sm_w));
        const uint64_t dx = kb::umma_desc_k_sw128(kb::smem_u32(sm_x));
        const uint32_t w_lo = static_cast<uint32_t>(dw), w_hi = static_cast<uint32_t>(dw >> 32);
        const uint32_t x_lo = static_cast<uint32_t>(dx), x_hi = static_cast<uint32_t>(dx >> 32);
        const uint32_t w_inc = static_cast<uint32_t>(p.w_slot) >> 4, x_inc = static_cast<uint32_t>(p.x_slot) >> 4;
        const uint32_t empty0 = kPair ? kb::map_to_cta(kb::smem_u32(empty), lead) : kb::smem_u32(empty);
        const uint32_t empty1 = kPair ? kb::map_to_cta(kb::smem_u32(empty), lead + 1u) : 0u;
        uint32_t s = 0, ph = 0, it = 0;
        bool ok = true;
        for (int pos = sched_id; pos < total_tiles; pos += sched_n, ++it) {
          const Tile t = tile_at(pos);
          const uint32_t idesc = idesc0 | (static_cast<uint32_t>(t.cols >> 3) << 17);
          if (!kb::mbar_wait_bounded(&tempty[it & 1u], ((it >> 1) & 1u) ^ 1u, p.limit_ns)) {
            kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_TEMPTY, (uint32_t)pos, 0);
            ok = false;
            break;
          }
          kb::tc_fence_after_sync();
          const uint32_t d = tmem_base + (it & 1u) * ACC_COLS;
          uint32_t accumulate = 0;
          for (int left = k1 - k0; left > 0; --left) {
            if (!kb::mbar_wait_bounded(&full[s], ph, p.limit_ns)) {
              kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_FULL, (uint32_t)pos, 0);
              ok = false;
              break;
            }
            kb::tc_fence_after_sync();
            const uint32_t sw = w_lo + s * w_inc, sx = x_lo + s * x_inc, bar = s * 8;
            if (++s == static_cast<uint32_t>(p.stages)) {
              s = 0;
              ph ^= 1u;
            }
            kb::umma_f16_x4<kPair>(d, sw, w_hi, sx, x_hi, W_STEP, X_STEP, idesc, accumulate);
            accumulate = 1;
            kb::umma_commit_warp<kPair>(empty0 + bar);
            if constexpr (kPair) kb::umma_commit_warp<kPair>(empty1 + bar);
          }
          if (!ok) break;
          const uint32_t f = kb::smem_u32(&tfull[it & 1u]);
          kb::umma_commit_warp<kPair>(kPair ? kb::map_to_cta(f, lead) : f);
          if constexpr (kPair) kb::umma_commit_warp<kPair>(kb::map_to_cta(f, lead + 1u));
        }
        if (!ok) *abort_flag = 1;
      }
      __syncwarp();
    } else if (warp >= 4 && p.split == 1) {
      // -------------------------------------------------------- epilogue ----
      // Warps q and q + 4 of the role drain lane quadrant q, 32 tokens in turn.
      const int q = warp & 3;
      const int turn = (warp - 4) >> 2;
      uint32_t it = 0;
      for (int pos = sched_id; pos < total_tiles; pos += sched_n, ++it) {
        const Tile t = tile_at(pos);
        const uint32_t acc = it & 1u;
        const int in_cta = q * 32 + lane;  // lane of the accumulator: output column of this CTA
        const int col0 = t.n0 + static_cast<int>(half) * w_cols;
        float bias = 0.0f;
        if (p.bias != nullptr && in_cta < w_cols && col0 + in_cta < p.N) bias = p.bias_scale * __bfloat162float(p.bias[col0 + in_cta]);
        const int vcol = q * 32 + (lane & ~3);  // first of the four columns this lane stores
        const bool col_ok = vcol < w_cols && col0 + vcol < p.N;
        const bool live = q * 32 < w_cols && col0 + q * 32 < p.N;
        const int last = live ? t.rows : 0;
        uint2 saved[8];
        if constexpr (kEpi == EPI_SLOPE) {
          // The saved values are on their way while the tile's products are made: a token per thread into the L2, this warp's first
          // tokens into registers.  Fetched when the accumulator was ready they took the last tile's epilogue 8 us.
          const int token = (warp - 4) * 32 + lane;
          if (token < t.rows && col0 < p.N) {
            kb::prefetch_l2(p.pre_in + static_cast<size_t>(t.row0 + token) * p.N + col0, static_cast<uint32_t>(min(w_cols, p.N - col0)) * 2);
          }
          if (turn * 32 < last) fetch_saved<16>(p, static_cast<size_t>(t.row0 + turn * 32) * p.N + col0 + vcol, t.rows - turn * 32, col_ok, lane, saved);
        }
        if (*abort_flag == 0 && !kb::mbar_wait_bounded(&tfull[acc], (it >> 1) & 1u, p.limit_ns, 2000)) {
          kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_TFULL, (uint32_t)pos, 0);
          *abort_flag = 1;
        }
        kb::tc_fence_after_sync();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * ACC_COLS;
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
        if (turn * 32 >= last) release();
#pragma unroll 1
        for (int c = turn * 32; c < last; c += 64) {
          const size_t at = static_cast<size_t>(t.row0 + c) * p.N + col0 + vcol;
          uint2 now[8];
          if constexpr (kEpi == EPI_SLOPE) {
#pragma unroll
            for (int i = 0; i < 8; ++i) now[i] = saved[i];
            if (c + 64 < last) fetch_saved<16>(p, at + static_cast<size_t>(64) * p.N, t.rows - c - 64, col_ok, lane, saved);
          }
          uint32_t r[32];
          kb::tmem_ld_32x32(taddr + c, r);
          kb::tmem_ld_wait();
          if (c + 64 >= last) release();
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
          finish<kEpi, 16>(p, f, bias, now, at, t.rows - c, col_ok, lane);
        }
      }
    } else if (warp == 4 && p.split > 1) {
      // The members of a cluster work on one tile each: wait here until this CTA's partial is complete.
      if (!kb::mbar_wait_bounded(&tfull[0], 0u, p.limit_ns, 1000)) {
        kb::report_status(p.status, KB_DEV_TIMEOUT_MBAR, kbl::SITE_TFULL, (uint32_t)sched_id, 0);
        *abort_flag = 1;
      }
      kb::tc_fence_before_sync();
    }
  }

  if constexpr (kKind == DENSE) {
    if (p.split > 1) {
      // --------------------------------------------- exchange of the partials ----
      // Chunk c of eight tokens belongs to member c * split / chunks.  Slot (chunk, source) of the owner's operand
      // ring holds 128 lanes x 8 tokens as [4 tokens][lane] float4: neighbouring lanes write neighbouring 16 bytes.
      __syncthreads();
      kb::cluster_sync_all();  // every member's MMAs have finished: all operand rings are free
      kb::tc_fence_after_sync();
      const Tile t = tile_at(sched_id);
      const int chunks = (t.rows + CHUNK - 1) / CHUNK;
      const int q = warp & 3;
      const int in_cta = q * 32 + lane;
      const int col0 = t.n0 + static_cast<int>(half) * w_cols;
      const bool live = q * 32 < w_cols && col0 + q * 32 < p.N;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
      constexpr int SLOT = LANES * CHUNK * 4;
      if (live) {
        for (int c = warp >> 2; c < chunks; c += THREADS / 128) {
          const int owner = c * p.split / chunks;
          if (owner == member) continue;
          const int first = (owner * chunks + p.split - 1) / p.split;  // the owner's first chunk
          const int src = member < owner ? member : member - 1;
          uint32_t r[8];
          kb::tmem_ld_32x8(taddr + c * CHUNK, r);
          kb::tmem_ld_wait();
          const uint32_t to = kb::map_to_cta(kb::smem_u32(base + ((c - first) * (p.split - 1) + src) * SLOT),
                                             static_cast<uint32_t>(owner) * (kPair ? 2u : 1u) + half);
#pragma unroll
          for (int i = 0; i < 2; ++i) kb::st_shared_cluster_v4(to + (i * LANES + in_cta) * 16, r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        }
      }
      float bias = 0.0f;
      if (p.bias != nullptr && in_cta < w_cols && col0 + in_cta < p.N) bias = p.bias_scale * __bfloat162float(p.bias[col0 + in_cta]);
      kb::cluster_sync_all();  // the partials are in place
      if (live) {
        const int vcol = q * 32 + (lane & ~3);
        const bool col_ok = vcol < w_cols && col0 + vcol < p.N;
        for (int c = warp >> 2; c < chunks; c += THREADS / 128) {
          if (c * p.split / chunks != member) continue;
          const int first = (member * chunks + p.split - 1) / p.split;
          const size_t at = static_cast<size_t>(t.row0 + c * CHUNK) * p.N + col0 + vcol;
          uint2 saved[2];
          if constexpr (kEpi == EPI_SLOPE) fetch_saved<4>(p, at, t.rows - c * CHUNK, col_ok, lane, saved);
          uint32_t r[8];
          kb::tmem_ld_32x8(taddr + c * CHUNK, r);
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = 0.f;
          const uint32_t from = kb::smem_u32(base) + in_cta * 16;
          kb::tmem_ld_wait();
#pragma unroll 1
          for (int m = 0; m < p.split; ++m) {  // ascending member order
            if (m == member) {
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] += __uint_as_float(r[i]);
            } else {
              const uint32_t slot = from + ((c - first) * (p.split - 1) + (m < member ? m : m - 1)) * SLOT;
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const float4 v = kb::ld_shared_v4(slot + i * LANES * 16);
                f[4 * i] += v.x; f[4 * i + 1] += v.y; f[4 * i + 2] += v.z; f[4 * i + 3] += v.w;
              }
            }
          }
          finish<kEpi, 4>(p, f, bias, saved, at, t.rows - c * CHUNK, col_ok, lane);
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

}  // namespace kbs
