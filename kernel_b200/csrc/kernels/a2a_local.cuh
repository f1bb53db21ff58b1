// The MoE round trip of a single rank: every expert is local, no row has to move.
//
// Included by a2a.cu inside its unnamed namespace, after a2a_dedup.cuh.
//
// With one rank the dispatch would copy a token's row into a receive region, the
// expert phase read it back and write a partial row, the combine read that: three
// passes over memory and two grid-wide hand-offs for values that depend on one row of x
// and k (expert, weight) pairs.  Here a CTA reads the row once, forms
//     out = sum_j  w_j * round(scale(e_j) * x)
// in fp32 in ascending j with the rounding points of the general kernels (the expert's
// output type, then the result's) and writes it once; outputs are equal to theirs bit
// for bit.  Bound by memory (x in, out out) for many tokens, by the launch for few.
// 7168 bf16 values, top-8, 256 experts: 2048 tokens 89 -> 13 us, one token 12 -> 3 us of GPU time.
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

constexpr int LOCAL_MAX_THREADS = 512;

// One CTA: one token and 1/splits of its row, kVecs 16-byte vectors per thread and step.
template <typename T, int kVecs>
__global__ void __launch_bounds__(LOCAL_MAX_THREADS) a2a_local_kernel(const A2aParams p, int splits) {
  __shared__ float s_scale[64], s_w[64];  // topk <= 64; a negative scale marks an expert id out of range
  const int t = blockIdx.x / splits;
  const int part = blockIdx.x - t * splits;
  const int per = (p.vecs + splits - 1) / splits;
  const int v0 = part * per, v1 = min(v0 + per, p.vecs);
  const int tid = threadIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(t) * p.row_bytes);
  uint4* dst = reinterpret_cast<uint4*>(p.out + static_cast<size_t>(t) * p.row_bytes);
  uint4 in[kVecs];
#pragma unroll
  for (int u = 0; u < kVecs; ++u) {
    const int v = v0 + tid + u * blockDim.x;
    if (v < v1) in[u] = kb::ld_nc_v4(src + v);
  }
  bool rounds = false;  // some scale differs from 1
  if (tid < p.k) {
    const int e = __ldg(p.idx + static_cast<size_t>(t) * p.k + tid);
    float scale = 1.0f;
    if (e < 0 || e >= p.E) {
      if (part == 0) kb::report_status(p.status, KB_DEV_BAD_INDEX, SITE_DISP_IDX, (uint32_t)(t * p.k + tid), p.epoch);
      scale = -1.0f;
    } else if (p.scale_mode == 2) {
      scale = static_cast<float>(e + 1) / static_cast<float>(p.E);
    }
    s_scale[tid] = scale;
    s_w[tid] = __ldg(p.w + static_cast<size_t>(t) * p.k + tid);
    rounds = scale != 1.0f;
  }
  rounds = __syncthreads_or(rounds);
  for (int vb = v0 + tid; vb < v1; vb += kVecs * blockDim.x) {
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
    for (int j = 0; j < p.k; ++j) {
      const float s = s_scale[j];
      if (s < 0.0f) continue;
      const uint64_t w2 = pack_f32x2(s_w[j], s_w[j]);
      if (rounds) {
        const uint64_t s2 = pack_f32x2(s, s);
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
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      const int v = vb + u * blockDim.x;
      float f[Vec16<T>::N];
#pragma unroll
      for (int i = 0; i < P; ++i) unpack_f32x2(acc[u][i], f[2 * i], f[2 * i + 1]);
      if (v < v1) dst[v] = Vec16<T>::store(f);
    }
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {  // rows longer than one step of the CTA
      const int v = vb + (kVecs + u) * blockDim.x;
      if (v < v1) in[u] = kb::ld_nc_v4(src + v);
    }
  }
}

template <typename T>
static int launch_local(const A2aParams& p, int sms, cudaStream_t st) {
  if (p.T == 0) return KB_OK;
  // Few tokens: one vector per thread and a row spread over CTAs of 128 threads, so that
  // every load is in flight at once; many: four vectors per thread, a row per CTA.
  const long long vecs = static_cast<long long>(p.T) * p.vecs;
  if (vecs < 4ll * 512 * sms) {
    const int splits = (p.vecs + 127) / 128;
    a2a_local_kernel<T, 1><<<p.T * splits, 128, 0, st>>>(p, splits);
  } else {
    int threads = ((p.vecs + 3) / 4 + 31) / 32 * 32;
    if (threads > LOCAL_MAX_THREADS) threads = LOCAL_MAX_THREADS;
    if (threads < 64) threads = 64;  // topk entries are fetched by the first 64 threads
    a2a_local_kernel<T, 4><<<p.T, threads, 0, st>>>(p, 1);
  }
  KB_CUDA_OK(cudaGetLastError());
  return KB_OK;
}
