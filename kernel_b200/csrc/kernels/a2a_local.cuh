// The MoE round trip of a single rank: every expert is local, no row has to move.
//
// Included by a2a.cu inside its unnamed namespace, after a2a_dedup.cuh.
//
// With one rank the dispatch would copy a token's row into a receive region, the
// expert phase read it back and write a partial row, the combine read that: three
// passes over memory and two grid-wide hand-offs for values that depend on one row of x
// and k (expert, weight) pairs.  Here a warp reads its part of the row once, forms
//     out = sum_j  w_j * round(scale(e_j) * x)
// in fp32 in ascending j with the rounding points of the general kernels (the expert's
// output type, then the result's) and writes it once; outputs are equal to theirs bit
// for bit.  Bound by memory (x in, out out) for many tokens, by the launch for few.
// 7168 bf16 values, top-8, 256 experts: 2048 tokens 89 -> 25 us a call, one token 12 -> 7 (3.6 us of GPU time).
//
// The arithmetic is next to the memory time (8 experts x 20 instructions per 16-byte
// vector), hence two values per instruction (f32x2) where the type allows.

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Rounds a pair of fp32 values to T and back.
template <typename T>
__device__ __forceinline__ uint64_t round_f32x2(uint64_t v);
template <>
__device__ __forceinline__ uint64_t round_f32x2<float>(uint64_t v) { return v; }
template <>
__device__ __forceinline__ uint64_t round_f32x2<__nv_bfloat16>(uint64_t v) {
  float lo, hi;
  unpack_f32x2(v, lo, hi);
  const uint32_t u = kb::pack_bf16x2(lo, hi);
  return pack_f32x2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
template <>
__device__ __forceinline__ uint64_t round_f32x2<__half>(uint64_t v) {
  float lo, hi;
  unpack_f32x2(v, lo, hi);
  const float2 f = __half22float2(__floats2half2_rn(lo, hi));
  return pack_f32x2(f.x, f.y);
}

constexpr int LOCAL_WARPS = 4;  // of a CTA

// A warp takes units of 32 * kVecs 16-byte vectors of one token's row, on its own: the (scale,
// weight) pairs of the token go through its share of shared memory, the next unit's row
// part and pairs are on their way while it computes.  (One CTA per row with a barrier between
// the pairs and the arithmetic left the latency of the loads exposed seven times in a row:
// 2048 tokens of 14 KB, bf16, 31 us.)
template <typename T, int kVecs, int kCtas>
__global__ void __launch_bounds__(32 * LOCAL_WARPS, kCtas) a2a_local_kernel(const A2aParams p, int parts, int units) {
  __shared__ float2 s_sw[LOCAL_WARPS][64];  // topk <= 64; a negative scale marks an expert id out of range
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* sw = s_sw[warp];
  const int stride = gridDim.x * LOCAL_WARPS;
  uint4 in[kVecs];
  int e[2];
  float w[2];
  auto fetch = [&](int unit) {
    const int t = unit / parts;
    const int v0 = (unit - t * parts) * (32 * kVecs) + lane;
    const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(t) * p.row_bytes);
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      if (v0 + 32 * u < p.vecs) in[u] = kb::ld_nc_v4(src + v0 + 32 * u);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (lane + 32 * i < p.k) {
        e[i] = __ldg(p.idx + static_cast<size_t>(t) * p.k + lane + 32 * i);
        w[i] = __ldg(p.w + static_cast<size_t>(t) * p.k + lane + 32 * i);
      }
    }
  };
  int unit = blockIdx.x * LOCAL_WARPS + warp;
  if (unit < units) fetch(unit);
  for (; unit < units; unit += stride) {
    const int t = unit / parts;
    const int part = unit - t * parts;
    bool differs = false;  // some scale is not 1
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (lane + 32 * i >= p.k) continue;
      float scale = 1.0f;
      if (e[i] < 0 || e[i] >= p.E) {
        if (part == 0) kb::report_status(p.status, KB_DEV_BAD_INDEX, SITE_DISP_IDX, (uint32_t)(t * p.k + lane + 32 * i), p.epoch);
        scale = -1.0f;
      } else if (p.scale_mode == 2) {
        scale = static_cast<float>(e[i] + 1) / static_cast<float>(p.E);
      }
      sw[lane + 32 * i] = make_float2(scale, w[i]);
      differs |= scale != 1.0f;
    }
    const bool rounds = __any_sync(0xffffffffu, differs);
    constexpr int P = Vec16<T>::N / 2;
    uint64_t xin[kVecs][P], acc[kVecs][P];
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      float f[Vec16<T>::N];
      Vec16<T>::load(in[u], f);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        xin[u][i] = pack_f32x2(f[2 * i], f[2 * i + 1]);
        acc[u][i] = 0ull;
      }
    }
    if (unit + stride < units) fetch(unit + stride);
    __syncwarp();
    for (int j = 0; j < p.k; ++j) {
      const float2 c = sw[j];
      if (c.x < 0.0f) continue;
      const uint64_t w2 = pack_f32x2(c.y, c.y);
      if (rounds) {
        const uint64_t s2 = pack_f32x2(c.x, c.x);
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
#pragma unroll
          for (int i = 0; i < P; ++i) acc[u][i] = fma_f32x2(w2, round_f32x2<T>(mul_f32x2(xin[u][i], s2)), acc[u][i]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < kVecs; ++u) {
#pragma unroll
          for (int i = 0; i < P; ++i) acc[u][i] = fma_f32x2(w2, xin[u][i], acc[u][i]);
        }
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(p.out + static_cast<size_t>(t) * p.row_bytes);
    const int v0 = part * (32 * kVecs) + lane;
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      float f[Vec16<T>::N];
#pragma unroll
      for (int i = 0; i < P; ++i) unpack_f32x2(acc[u][i], f[2 * i], f[2 * i + 1]);
      if (v0 + 32 * u < p.vecs) dst[v0 + 32 * u] = Vec16<T>::store(f);
    }
    __syncwarp();  // the pairs may be overwritten
  }
}

template <typename T, int kVecs, int kCtas>
static int launch_local_as(const A2aParams& p, int sms, cudaStream_t st) {
  const int parts = (p.vecs + 32 * kVecs - 1) / (32 * kVecs);
  const long long units = static_cast<long long>(p.T) * parts;
  if (units > 0x3fffffff) return KB_ERR_UNSUPPORTED;  // three launches of the general kernels
  // as many rounds as the resident warps need, all warps with the same number of units
  const long long resident = static_cast<long long>(sms) * kCtas * LOCAL_WARPS;
  const long long per_cta = (units + resident - 1) / resident * LOCAL_WARPS;
  const int grid = static_cast<int>((units + per_cta - 1) / per_cta);
  a2a_local_kernel<T, kVecs, kCtas><<<grid, 32 * LOCAL_WARPS, 0, st>>>(p, parts, static_cast<int>(units));
  KB_CUDA_OK(cudaGetLastError());
  return KB_OK;
}

template <typename T>
static int launch_local(const A2aParams& p, int sms, cudaStream_t st) {
  if (p.T == 0) return KB_OK;
  // Few tokens: one vector per lane spreads a row over more warps (up to about 80 tokens of
  // 14 KB).  Many: what fits the registers without giving up resident warps; fp32 has
  // half the values per vector, so twice the vectors (2048 tokens of 7168 values: bf16 31.0 -> 26.9 us, with unit scales
  // 22.8 -> 16.7; fp32 30.8 -> 24.9; 1500 tokens of 5000 bf16 values are unchanged at 16.5).
  if (static_cast<long long>(p.T) * p.vecs < 16ll * 32 * sms) return launch_local_as<T, 1, 8>(p, sms, st);
  if constexpr (sizeof(T) == 4) return launch_local_as<T, 4, 4>(p, sms, st);
  else return launch_local_as<T, 2, 8>(p, sms, st);
}
