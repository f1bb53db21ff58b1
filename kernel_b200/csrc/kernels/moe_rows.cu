// Row movement of a MoE layer whose experts are all on this GPU (one rank):
//
//   permute    token rows -> expert-major rows (one copy per (token, choice)), with the group table the
//              grouped GEMMs read (gemm_local.cuh); nothing goes through the host
//   combine    out[t] = sum_j w[t, j] * Y[row(t, j)], fp32 in ascending j
//   grad_rows  backward of combine: dY[row(t, j)] = w[t, j] * dy[t] and dw[t, j] = <dy[t], Y[row(t, j)]>
//
// All three are bound by memory: every row is read and written once with 16-byte
// accesses.  The slot of a (token, choice) copy is computed as in the dispatch kernel
// (a2a.cu): every CTA histograms the whole routing table (it fits the L2 and is at
// most a few hundred KB), so no count exchange, atomics across CTAs or second launch is
// needed, and rows of an expert are in token order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <string.h>

#include <initializer_list>

#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../include/kb200.h"

namespace {

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;
constexpr int PERM_THREADS = 512;
constexpr int PERM_WARPS = PERM_THREADS / 32;
constexpr int PERM_VECS = 2;     // 16-byte vectors per lane of one copy task: 1 KB of a row
constexpr int HIST = 16;         // table entries a thread keeps in flight
constexpr int MAX_EXPERTS = 1024;
constexpr int MAX_ENT = 1024;  // (token, choice) entries of one CTA of the permute kernel

enum Site : uint32_t { SITE_MOE_IDX = 41 };

struct MoeParams {
  int T, k, E, vecs;  // vecs: 16-byte vectors of a row
  int pad;            // rows of an expert start at, and are zero-filled up to, multiples of this
  int tok_per_cta;
  const int32_t* idx;
  const uint4* x;
  uint4* rows;
  int32_t* slots;      // [T][k] row of a copy, or -1 (expert id out of range)
  int32_t* row_start;  // [E]
  int32_t* row_count;  // [E] rows, padding not counted
  int32_t* row_padded; // [E] rows, padding counted
  uint32_t* status;
};

__device__ __forceinline__ void load8(const uint4& u, float* f) {
  float2 t;
  t = kb::unpack_bf16x2(u.x); f[0] = t.x; f[1] = t.y;
  t = kb::unpack_bf16x2(u.y); f[2] = t.x; f[3] = t.y;
  t = kb::unpack_bf16x2(u.z); f[4] = t.x; f[5] = t.y;
  t = kb::unpack_bf16x2(u.w); f[6] = t.x; f[7] = t.y;
}
__device__ __forceinline__ uint4 store8(const float* f) {
  return make_uint4(kb::pack_bf16x2(f[0], f[1]), kb::pack_bf16x2(f[2], f[3]), kb::pack_bf16x2(f[4], f[5]), kb::pack_bf16x2(f[6], f[7]));
}

// Bound by latency up to some thousand rows: the routing table, the ranking and the rows
// follow one another.  So the first rows are fetched before the table, the table in
// one round of loads where it fits, and an entry costs one shared-memory atomic (it is
// counted either before or after this CTA's first).  1024 tokens of 4 KB, top-8 of 64
// experts, cold caches: 17.2 -> 13.9 us (46 MB, 7 us at the copy rate).
__global__ void __launch_bounds__(PERM_THREADS) moe_permute_kernel(const MoeParams p) {
  // entries of an expert: from this CTA's first token on (later: all of them), and before it
  __shared__ int32_t tot[MAX_EXPERTS], pre[MAX_EXPERTS];
  __shared__ int32_t start[MAX_EXPERTS];
  __shared__ int32_t ent_e[MAX_ENT], ent_slot[MAX_ENT];
  __shared__ int32_t s_warp[PERM_WARPS];
  kb::wait_for_previous_launch();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = min(static_cast<int>(blockIdx.x) * p.tok_per_cta, p.T);
  const int t1 = min(t0 + p.tok_per_cta, p.T);
  const int n_ent = (t1 - t0) * p.k;
  const int total = p.T * p.k;
  // a copy task: 32 * PERM_VECS vectors of one token's row, fetched once and written k times
  const int chunks = (p.vecs + 32 * PERM_VECS - 1) / (32 * PERM_VECS);
  const int tasks = (t1 - t0) * chunks;
  uint4 val[PERM_VECS];
  auto fetch = [&](int c) {
    const int i = c / chunks;
    const int v0 = (c - i * chunks) * (32 * PERM_VECS) + lane;
    const uint4* src = p.x + static_cast<size_t>(t0 + i) * p.vecs;
#pragma unroll
    for (int u = 0; u < PERM_VECS; ++u) {
      if (v0 + u * 32 < p.vecs) val[u] = kb::ld_stream_v4(src + v0 + u * 32);
    }
  };
  if (warp < tasks) fetch(warp);
  for (int i = tid; i < n_ent; i += PERM_THREADS) ent_e[i] = p.idx[t0 * p.k + i];
  for (int e = tid; e < p.E; e += PERM_THREADS) tot[e] = pre[e] = 0;
  __syncthreads();
  for (int i0 = tid; i0 < total; i0 += HIST * PERM_THREADS) {  // all fetched before any is counted
    int ev[HIST];
#pragma unroll
    for (int u = 0; u < HIST; ++u) ev[u] = i0 + u * PERM_THREADS < total ? p.idx[i0 + u * PERM_THREADS] : 0;
#pragma unroll
    for (int u = 0; u < HIST; ++u) {
      const int i = i0 + u * PERM_THREADS;
      if (i >= total) continue;
      if (ev[u] < 0 || ev[u] >= p.E) {
        if (blockIdx.x == 0) kb::report_status(p.status, KB_DEV_BAD_INDEX, SITE_MOE_IDX, (uint32_t)i, 0);
        continue;
      }
      atomicAdd(i < t0 * p.k ? &pre[ev[u]] : &tot[ev[u]], 1);
    }
  }
  __syncthreads();
  {  // exclusive prefix of the padded counts
    constexpr int PER = MAX_EXPERTS / PERM_THREADS;
    int v[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = tid * PER + j;
      if (e < p.E) tot[e] += pre[e];
      v[j] = e < p.E ? (tot[e] + p.pad - 1) / p.pad * p.pad : 0;
      sum += v[j];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int i = 0; i < warp; ++i) run += s_warp[i];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = tid * PER + j;
      if (e < p.E) {
        start[e] = run;
        if (blockIdx.x == 0) {
          p.row_start[e] = run;
          p.row_count[e] = tot[e];
          p.row_padded[e] = v[j];
        }
      }
      run += v[j];
    }
  }
  __syncthreads();
  for (int i = tid; i < n_ent; i += PERM_THREADS) {
    const int e = ent_e[i];
    int slot = -1;
    if (e >= 0 && e < p.E) {
      int r = 0;
      for (int j = 0; j < i; ++j) r += ent_e[j] == e ? 1 : 0;
      slot = start[e] + pre[e] + r;
    }
    ent_slot[i] = slot;
    p.slots[t0 * p.k + i] = slot;
  }
  __syncthreads();
  for (int c = warp; c < tasks; c += PERM_WARPS) {
    const int i = c / chunks;
    const int v0 = (c - i * chunks) * (32 * PERM_VECS) + lane;
    if (c != warp) fetch(c);
    for (int j = 0; j < p.k; ++j) {
      const int slot = ent_slot[i * p.k + j];
      if (slot < 0) continue;
      uint4* dst = p.rows + static_cast<size_t>(slot) * p.vecs;
#pragma unroll
      for (int u = 0; u < PERM_VECS; ++u) {
        if (v0 + u * 32 < p.vecs) dst[v0 + u * 32] = val[u];
      }
    }
  }
  if (p.pad > 1) {  // rows between an expert's last one and the next multiple of pad, a quarter of an expert's per CTA
    for (int u = blockIdx.x; u < 4 * p.E; u += gridDim.x) {
      const int e = u >> 2;
      const int r1 = (tot[e] + p.pad - 1) / p.pad * p.pad;
      uint4* dst = p.rows + static_cast<size_t>(start[e] + tot[e]) * p.vecs;
      const int n = (r1 - tot[e]) * p.vecs;
      for (int v = (u & 3) * PERM_THREADS + tid; v < n; v += 4 * PERM_THREADS) dst[v] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

struct CombineParams {
  int T, k, vecs, splits;
  const uint4* y;
  const int32_t* slots;
  const float* w;  // null: unit weights
  uint4* out;
};

// One CTA: one token and 1/splits of its row; a thread keeps eight rows' loads in flight.
__global__ void __launch_bounds__(128) moe_combine_kernel(const CombineParams p) {
  kb::wait_for_previous_launch();
  const int t = blockIdx.x / p.splits;
  const int part = blockIdx.x - t * p.splits;
  const int per = (p.vecs + p.splits - 1) / p.splits;
  const int v1 = min((part + 1) * per, p.vecs);
  const int32_t* ts = p.slots + static_cast<size_t>(t) * p.k;
  for (int v = part * per + static_cast<int>(threadIdx.x); v < v1; v += 128) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int j0 = 0; j0 < p.k; j0 += 8) {
      uint4 u[8];
      float wj[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        u[j] = make_uint4(0u, 0u, 0u, 0u);
        wj[j] = 0.f;
        if (j0 + j < p.k) {
          const int s = ts[j0 + j];
          if (s >= 0) {
            u[j] = kb::ld_global_v4(p.y + static_cast<size_t>(s) * p.vecs + v);
            wj[j] = p.w != nullptr ? p.w[static_cast<size_t>(t) * p.k + j0 + j] : 1.f;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float f[8];
        load8(u[j], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(wj[j], f[i], acc[i]);
      }
    }
    p.out[static_cast<size_t>(t) * p.vecs + v] = store8(acc);
  }
}

struct GradParams {
  int T, k, E, vecs;
  const uint4* dy;
  const uint4* y;
  const int32_t* slots;
  const float* w;
  uint4* dyr;
  float* dw;
  const int32_t *row_start, *row_count, *row_padded;
};

// One CTA per token; the CTAs behind the last token zero-fill the padding rows of dyr, four
// per expert (one: 17.7 us for 1024 tokens of 4 KB, top-8 of 64; four: 14.0).
__global__ void __launch_bounds__(THREADS) moe_grad_rows_kernel(const GradParams p) {
  kb::wait_for_previous_launch();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (static_cast<int>(blockIdx.x) >= p.T) {
    for (int u = blockIdx.x - p.T; u < 4 * p.E; u += gridDim.x - p.T) {
      const int e = u >> 2;
      const int first = p.row_start[e] + p.row_count[e];
      const int n = (p.row_padded[e] - p.row_count[e]) * p.vecs;
      for (int v = (u & 3) * THREADS + tid; v < n; v += 4 * THREADS) p.dyr[static_cast<size_t>(first) * p.vecs + v] = make_uint4(0u, 0u, 0u, 0u);
    }
    return;
  }
  // A warp takes whole (token, choice) rows: no reduction across warps.
  const int t = blockIdx.x;
  const uint4* dy = p.dy + static_cast<size_t>(t) * p.vecs;
  for (int j = warp; j < p.k; j += WARPS) {
    const int s = p.slots[static_cast<size_t>(t) * p.k + j];
    float dot = 0.f;
    if (s >= 0) {
      const float wj = p.w[static_cast<size_t>(t) * p.k + j];
      const uint4* y = p.y + static_cast<size_t>(s) * p.vecs;
      uint4* out = p.dyr + static_cast<size_t>(s) * p.vecs;
      for (int v0 = lane; v0 < p.vecs; v0 += 128) {
        uint4 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (v0 + 32 * u < p.vecs) {
            a[u] = kb::ld_global_v4(dy + v0 + 32 * u);
            b[u] = kb::ld_stream_v4(y + v0 + 32 * u);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (v0 + 32 * u >= p.vecs) continue;
          float f[8], g[8];
          load8(a[u], f);
          load8(b[u], g);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            dot = fmaf(f[i], g[i], dot);
            f[i] *= wj;
          }
          out[v0 + 32 * u] = store8(f);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == 0) p.dw[static_cast<size_t>(t) * p.k + j] = dot;
  }
}

int sm_count(int* sms) {
  static int cached[64] = {0};
  int dev = 0;
  KB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && cached[dev] > 0) {
    *sms = cached[dev];
    return KB_OK;
  }
  KB_CUDA_OK(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
  if (dev >= 0 && dev < 64) cached[dev] = *sms;
  return KB_OK;
}

int check_sizes(int T, int k, int E, int hidden) {
  if (T < 0 || k < 1 || k > 64 || E < 1 || E > MAX_EXPERTS || hidden < 8 || hidden % 8 != 0 || static_cast<long long>(T) * k > (1 << 28)) {
    kb::set_error("moe rows: T=%d k=%d experts=%d hidden=%d out of range (hidden a multiple of 8)", T, k, E, hidden);
    return KB_ERR_ARG;
  }
  return KB_OK;
}

// Rows are moved in 16-byte vectors, tables and weights in 4-byte words.
int check_pointers(std::initializer_list<const void*> rows, std::initializer_list<const void*> words) {
  for (const void* q : rows) {
    if ((reinterpret_cast<uintptr_t>(q) & 15u) != 0) {
      kb::set_error("moe rows: row buffers must be 16-byte aligned");
      return KB_ERR_ARG;
    }
  }
  for (const void* q : words) {
    if ((reinterpret_cast<uintptr_t>(q) & 3u) != 0) {
      kb::set_error("moe rows: tables and weights must be 4-byte aligned");
      return KB_ERR_ARG;
    }
  }
  return KB_OK;
}

}  // namespace

extern "C" int kb_moe_permute(const void* x, const int32_t* indices, int T, int k, int experts, int hidden, int pad, void* rows,
                              int32_t* slots, int32_t* row_start, int32_t* row_count, int32_t* row_padded, uint32_t* status,
                              void* stream) {
  int rc = check_sizes(T, k, experts, hidden);
  if (rc != KB_OK) return rc;
  if (pad < 1) return KB_ERR_ARG;
  rc = check_pointers({x, rows}, {indices, slots, row_start, row_count, row_padded});
  if (rc != KB_OK) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc != KB_OK) return rc;
  MoeParams p;
  p.T = T;
  p.k = k;
  p.E = experts;
  p.vecs = hidden / 8;
  p.pad = pad;
  p.idx = indices;
  p.x = static_cast<const uint4*>(x);
  p.rows = static_cast<uint4*>(rows);
  p.slots = slots;
  p.row_start = row_start;
  p.row_count = row_count;
  p.row_padded = row_padded;
  p.status = status;
  // Every CTA reads the whole table: no more CTAs than fill the chip, as long as a
  // CTA's entries fit its ranking buffer.
  int per = (T + 2 * sms - 1) / (2 * sms);
  if (per < 1) per = 1;
  if (per > MAX_ENT / k) per = MAX_ENT / k;
  p.tok_per_cta = per;
  const int grid = T > 0 ? (T + per - 1) / per : 1;
  KB_CUDA_OK(kb::launch_after(moe_permute_kernel, grid, PERM_THREADS, stream, p));
  return KB_OK;
}

extern "C" int kb_moe_combine(const void* y, const int32_t* slots, const float* weights, int T, int k, int hidden, void* out, void* stream) {
  int rc = check_sizes(T, k, 1, hidden);
  if (rc != KB_OK || T == 0) return rc;
  rc = check_pointers({y, out}, {slots, weights});
  if (rc != KB_OK) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc != KB_OK) return rc;
  CombineParams p = {T, k, hidden / 8, 1, static_cast<const uint4*>(y), slots, weights, static_cast<uint4*>(out)};
  while (T * p.splits < 4 * sms && p.vecs > 32 * p.splits) p.splits *= 2;  // few tokens: spread a row over several CTAs
  KB_CUDA_OK(kb::launch_after(moe_combine_kernel, T * p.splits, 128, stream, p));
  return KB_OK;
}

extern "C" int kb_moe_grad_rows(const void* dy, const void* y, const int32_t* slots, const float* weights, int T, int k, int experts,
                                int hidden, void* dyr, float* dw, const int32_t* row_start, const int32_t* row_count,
                                const int32_t* row_padded, void* stream) {
  int rc = check_sizes(T, k, experts, hidden);
  if (rc != KB_OK) return rc;
  rc = check_pointers({dy, y, dyr}, {slots, weights, dw});
  if (rc != KB_OK) return rc;
  GradParams p = {T, k, experts, hidden / 8, static_cast<const uint4*>(dy), static_cast<const uint4*>(y), slots, weights,
                  static_cast<uint4*>(dyr), dw, row_start, row_count, row_padded};
  KB_CUDA_OK(kb::launch_after(moe_grad_rows_kernel, T + 4 * (experts < 64 ? experts : 64), THREADS, stream, p));
  return KB_OK;
}
