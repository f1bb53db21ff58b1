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
// output type, then the result's) and writes it once; outputs are equal to theirs value
// for value.  Bound by memory (x in, out out) for many tokens, by the launch for few.
// 7168 bf16 values, top-8, 256 experts: 2048 tokens 89 -> 16.1 us, one token 12 -> 7 a call (1.5 us of GPU time).
//
// The arithmetic is next to the memory time (8 experts x 16 instructions per 16-byte vector, 6.5 us of issue slots;
// 9.0 us to read and write the rows at the copy rate), hence two values per instruction, in fp32 (f32x2) and for the
// scaling in the element type itself.

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

// Products of a pair in T itself.  Where the scale is a value of T this is one instruction for the product in fp32
// and its rounding: a product of two 16-bit values has at most 22 significant bits and, with a scale of at least 1/1024,
// no digit below the smallest fp32 value, so fp32 holds it exactly and both forms round the same number once.
template <typename T>
__device__ __forceinline__ uint32_t mul_t2(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t mul_t2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <>
__device__ __forceinline__ uint32_t mul_t2<__half>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <typename T>
__device__ __forceinline__ uint32_t both_t2(float v);  // v in both halves
template <>
__device__ __forceinline__ uint32_t both_t2<__nv_bfloat16>(float v) { return kb::pack_bf16x2(v, v); }
template <>
__device__ __forceinline__ uint32_t both_t2<__half>(float v) {
  const __half2 h = __floats2half2_rn(v, v);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T>
__device__ __forceinline__ uint64_t widen_t2(uint32_t u);  // as a pair of fp32 values
template <>
__device__ __forceinline__ uint64_t widen_t2<__nv_bfloat16>(uint32_t u) {
  // A byte permutation: a shift becomes a multiplication on the pipe that multiplies and adds already (16.6 -> 15.7 us).
  uint32_t lo;
  asm("prmt.b32 %0, %1, 0, 0x1044;" : "=r"(lo) : "r"(u));
  return pack_f32x2(__uint_as_float(lo), __uint_as_float(u & 0xffff0000u));
}
template <>
__device__ __forceinline__ uint64_t widen_t2<__half>(uint32_t u) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
  return pack_f32x2(f.x, f.y);
}
// Whether a scale is a value of T.
template <typename T>
__device__ __forceinline__ bool is_value_of(float v) {
  if constexpr (sizeof(T) == 4) return true;
  else {
    float lo, hi;
    unpack_f32x2(widen_t2<T>(both_t2<T>(v)), lo, hi);
    return lo == v;
  }
}

constexpr int LOCAL_WARPS = 4;  // of a CTA

// What is known of the experts' scales before the launch: all are 1, all are values of T, nothing.  Each has a kernel of its own: with
// the three loops in one, registers and schedule were those of the widest.  2048 tokens of 7168 bf16 values, top-8, inputs and outputs out of
// the L2: scales of 1 14.7 -> 11.6 us (9.0 at the copy rate), exact ones 17.3 -> 16.2, others 23.1 -> 22.9.
enum Scales { UNIT, EXACT, ANY };
// (e + 1) / E for all e: a power of two divides exactly, and e + 1 has the digits of T (8 of bf16, 11 of fp16)
template <typename T>
static bool exact_scales(int E) {
  return (E & (E - 1)) == 0 && E <= (std::is_same<T, __half>::value ? 1024 : 256);
}

// What a warp needs of one (token, choice): the routing weight twice, as an operand of the two-value instructions, and the
// expert's scale as fp32 and as a pair of T.
struct alignas(16) LocalChoice {
  float w0, w1;
  uint32_t scale2;
  float scale;
};

// A warp takes a fixed part of the rows, 32 * kVecs 16-byte vectors, of every `step`-th token, on its own: the
// choices of a token go through its share of shared memory, the next token's row part and choices are on their way while it
// computes.  Issue slots are what bounds it (52 % of them at unit scales, 58 % with scales, at 37 % of the copy rate, in the
// form before this one), so nothing is done per choice that can be done per token: entries out of range are left out
// of the list instead of being skipped in the loop, operands are stored the way the instructions want them, and
// parts that stay the same need no division.
template <typename T, int kVecs, int kCtas, Scales kScales>
__global__ void __launch_bounds__(32 * LOCAL_WARPS, kCtas) a2a_local_kernel(const A2aParams p, int parts, int step) {
  __shared__ LocalChoice s_choice[LOCAL_WARPS][64];  // topk <= 64
  kb::wait_for_previous_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = blockIdx.x * LOCAL_WARPS + warp;
  int t = gw / parts;
  if (t >= step) return;
  const int part = gw - t * parts;
  LocalChoice* choice = s_choice[warp];
  const int v0 = part * (32 * kVecs) + lane;
  const bool whole = (part + 1) * (32 * kVecs) <= p.vecs;
  const uint4* src = reinterpret_cast<const uint4*>(p.x) + v0;
  uint4* dst = reinterpret_cast<uint4*>(p.out) + v0;
  uint4 in[kVecs];
  int e[2];
  float w[2];
  auto fetch = [&](int at) {
    const uint4* row = src + static_cast<size_t>(at) * p.vecs;
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      if (whole || v0 + 32 * u < p.vecs) in[u] = kb::ld_stream_v4(row + 32 * u);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (lane + 32 * i < p.k) {
        e[i] = p.idx[static_cast<size_t>(at) * p.k + lane + 32 * i];
        w[i] = p.w[static_cast<size_t>(at) * p.k + lane + 32 * i];
      }
    }
  };
#pragma unroll
  for (int u = 0; u < kVecs; ++u) in[u] = make_uint4(0u, 0u, 0u, 0u);
  if (t < p.T) fetch(t);
  for (; t < p.T; t += step) {
    bool differs = false, inexact = false;  // some scale is not 1, not a value of T
    int n = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (32 * i >= p.k) break;
      const bool mine = lane + 32 * i < p.k;
      const bool valid = mine && e[i] >= 0 && e[i] < p.E;
      if (mine && !valid && part == 0) kb::report_status(p.status, KB_DEV_BAD_INDEX, SITE_DISP_IDX, (uint32_t)(t * p.k + lane + 32 * i), p.epoch);
      const float scale = kScales != UNIT && valid ? static_cast<float>(e[i] + 1) / static_cast<float>(p.E) : 1.0f;
      const uint32_t all = __ballot_sync(0xffffffffu, valid);
      if (valid) {
        LocalChoice c;
        c.w0 = c.w1 = w[i];
        c.scale2 = 0u;
        if constexpr (sizeof(T) == 2) c.scale2 = both_t2<T>(scale);
        c.scale = scale;
        choice[n + __popc(all & ((1u << lane) - 1u))] = c;
        differs |= scale != 1.0f;
        inexact |= !is_value_of<T>(scale);
      }
      n += __popc(all);
    }
    const bool rounds = kScales == EXACT || (kScales == ANY && __any_sync(0xffffffffu, differs));
    const bool exact = kScales == EXACT || (kScales == ANY && !__any_sync(0xffffffffu, inexact));
    constexpr int P = Vec16<T>::N / 2;
    uint64_t acc[kVecs][P];
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
#pragma unroll
      for (int i = 0; i < P; ++i) acc[u][i] = 0ull;
    }
    if (kScales != UNIT && sizeof(T) == 2 && rounds && exact) {
      if constexpr (kScales != UNIT && sizeof(T) == 2) {
        uint32_t xin[kVecs][P];
#pragma unroll
        for (int u = 0; u < kVecs; ++u) xin[u][0] = in[u].x, xin[u][1] = in[u].y, xin[u][2] = in[u].z, xin[u][3] = in[u].w;
        if (t + step < p.T) fetch(t + step);
        __syncwarp();
#pragma unroll 8
        for (int j = 0; j < n; ++j) {
          const LocalChoice c = choice[j];
          const uint64_t w2 = pack_f32x2(c.w0, c.w1);
#pragma unroll
          for (int u = 0; u < kVecs; ++u) {
#pragma unroll
            for (int i = 0; i < P; ++i) acc[u][i] = fma_f32x2(w2, widen_t2<T>(mul_t2<T>(xin[u][i], c.scale2)), acc[u][i]);
          }
        }
      }
    } else if constexpr (kScales != EXACT) {
      uint64_t xin[kVecs][P];
#pragma unroll
      for (int u = 0; u < kVecs; ++u) {
        float f[Vec16<T>::N];
        Vec16<T>::load(in[u], f);
#pragma unroll
        for (int i = 0; i < P; ++i) xin[u][i] = pack_f32x2(f[2 * i], f[2 * i + 1]);
      }
      if (t + step < p.T) fetch(t + step);
      __syncwarp();
      if (kScales == ANY && rounds) {
#pragma unroll 2
        for (int j = 0; j < n; ++j) {
          const LocalChoice c = choice[j];
          const uint64_t w2 = pack_f32x2(c.w0, c.w1), s2 = pack_f32x2(c.scale, c.scale);
#pragma unroll
          for (int u = 0; u < kVecs; ++u) {
#pragma unroll
            for (int i = 0; i < P; ++i) acc[u][i] = fma_f32x2(w2, round_f32x2<T>(mul_f32x2(xin[u][i], s2)), acc[u][i]);
          }
        }
      } else {
#pragma unroll 4
        for (int j = 0; j < n; ++j) {
          const uint64_t w2 = pack_f32x2(choice[j].w0, choice[j].w1);
#pragma unroll
          for (int u = 0; u < kVecs; ++u) {
#pragma unroll
            for (int i = 0; i < P; ++i) acc[u][i] = fma_f32x2(w2, xin[u][i], acc[u][i]);
          }
        }
      }
    }
    uint4* row = dst + static_cast<size_t>(t) * p.vecs;
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      float f[Vec16<T>::N];
#pragma unroll
      for (int i = 0; i < P; ++i) unpack_f32x2(acc[u][i], f[2 * i], f[2 * i + 1]);
      if (whole || v0 + 32 * u < p.vecs) row[32 * u] = Vec16<T>::store(f);
    }
    __syncwarp();  // the choices may be overwritten
  }
}

// Resident CTAs of an SM by vectors per lane: what the registers allow.  fp32 rows have half the values per vector and need no widening:
// five instead of four 21.7 -> 19.2 us with scales, 17.4 -> 15.7 without (2048 tokens of 7168, top-8 and top-6).
constexpr int local_ctas(int vecs, int elem_bytes) { return vecs == 1 ? 8 : vecs == 2 ? 6 : elem_bytes == 4 ? 5 : 4; }

template <typename T, int kVecs>
static int launch_local_as(const A2aParams& p, int sms, cudaStream_t st) {
  constexpr int kCtas = local_ctas(kVecs, sizeof(T));
  const int parts = (p.vecs + 32 * kVecs - 1) / (32 * kVecs);
  const long long units = static_cast<long long>(p.T) * parts;
  if (units > 0x3fffffff) return KB_ERR_UNSUPPORTED;  // three launches of the general kernels
  // All resident warps, though some then have a token more than others: as many warps as have the same number left
  // every seventh SM a CTA short (2048 tokens of 14 KB 18.6 us against 16.8).
  const long long resident = static_cast<long long>(sms) * kCtas * LOCAL_WARPS;
  const long long at_once = resident < parts ? 1 : resident / parts;  // tokens
  const long long step = at_once < p.T ? at_once : p.T;
  const int grid = static_cast<int>((step * parts + LOCAL_WARPS - 1) / LOCAL_WARPS);
  auto* kernel = p.scale_mode == 2 ? a2a_local_kernel<T, kVecs, kCtas, ANY> : a2a_local_kernel<T, kVecs, kCtas, UNIT>;
  if constexpr (sizeof(T) == 2) {
    if (p.scale_mode == 2 && exact_scales<T>(p.E)) kernel = a2a_local_kernel<T, kVecs, kCtas, EXACT>;
  }
  KB_CUDA_OK(kb::launch_after(kernel, grid, 32 * LOCAL_WARPS, st, p, parts, static_cast<int>(step)));
  return KB_OK;
}

// Vectors per lane.  Few tokens: one, which spreads a row over more warps (64 tokens of 14 KB 1.94 us of GPU time against 2.05
// with four, 128 tokens 2.95 and 2.60: the line is at about 60).  Many: four, which do with the fewest instructions per value
// what the registers allow; back to back in a graph, three inputs and outputs in turn, 7168 values, top-8, us with 1 / 2 / 4 vectors:
//   2048 tokens bf16, scales exact  21.9 17.6 16.2    unit scales 17.2 12.7 11.6    scales not bf16 values 28.1 23.8 22.9
//   2048 tokens fp16, exact         23.7 19.9 19.0    fp32 41.1  -   20.7           256 tokens bf16, exact  4.3  3.7  3.7
// In between a wide form may need a round of the resident warps more for a few tokens, leave most of a row's last warp idle
// or fill the SMs unevenly, so 16-bit rows count the rounds and the CTAs of an SM: bf16, scales not bf16 values, 1 / 2 / 4 vectors
//   700 tokens of 1048   3.4  3.7  4.2    300 of 4104   4.0  3.8  4.3    2048 of 2056   6.9  5.8  6.5    2048 of 2560   9.8  8.1  9.5
// The constants were fitted when one kernel had all three kinds of scale.  Over 68 cases of each kind past the first line (64 to 2048
// tokens of 1024 to 7168 16-bit values) the pick is 1.8 % above the best form on average with exact scales, 1.5 with others and 3.5 with
// scales of 1; always four 8.3, 9.1 and 2.1.
inline int local_vecs(int tokens, int vecs, int elem_bytes, int sms) {
  const long long all = static_cast<long long>(tokens) * vecs;
  if (elem_bytes == 4) return all < 16ll * 32 * sms ? 1 : 4;
  if (all < 12ll * 32 * sms) return 1;
  int best = 1;
  double best_cost = 1e30;
  for (int v = 1; v <= 4; v *= 2) {
    const int parts = (vecs + 32 * v - 1) / (32 * v);
    const long long at_once = static_cast<long long>(sms) * local_ctas(v, elem_bytes) * LOCAL_WARPS / parts;  // tokens
    const long long step = at_once < 1 ? 1 : at_once < tokens ? at_once : tokens;
    const double per_sm = static_cast<double>(((step * parts + LOCAL_WARPS - 1) / LOCAL_WARPS + sms - 1) / sms);  // CTAs
    const double rounds = static_cast<double>((tokens + step - 1) / step) + 2.6 * tokens / step;
    const double cost = rounds * (per_sm * (v + 0.13) + 1.5) + (v == 1 ? 1.8 : v == 2 ? -3.4 : 0.0);
    if (cost < best_cost) {
      best_cost = cost;
      best = v;
    }
  }
  return best;
}

template <typename T>
static int launch_local(const A2aParams& p, int sms, cudaStream_t st) {
  if (p.T == 0) return KB_OK;
  switch (local_vecs(p.T, p.vecs, sizeof(T), sms)) {
    case 1: return launch_local_as<T, 1>(p, sms, st);
    case 2:
      if constexpr (sizeof(T) == 2) return launch_local_as<T, 2>(p, sms, st);
  }
  return launch_local_as<T, 4>(p, sms, st);
}
