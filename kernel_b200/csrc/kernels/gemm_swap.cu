// Host side of the products with exchanged operands (device code: gemm_swap.cuh).
#include "gemm_swap.cuh"

#include <math.h>
#include <string.h>

#include "gemm_local_host.h"
#include "gemm_swap.h"

namespace {

using namespace kbs;
using kbl::ceil_div;

template <Kind kKind, bool kWMn, Epi kEpi>
const void* kernel_of(bool pair) {
  return pair ? (const void*)gemm_swap_kernel<kKind, true, kWMn, kEpi> : (const void*)gemm_swap_kernel<kKind, false, kWMn, kEpi>;
}

// An activation follows a product whose weights are contiguous along K (forward), a slope one
// whose weights are contiguous along N (backward).
const void* find_kernel(int kind, bool w_mn, int epi, bool pair, int* row) {
  *row = (kind == KB_LOCAL_ROWS ? 4 : 0) + (w_mn ? 2 : 0) + (epi != EPI_PLAIN ? 1 : 0);
  if (epi != EPI_PLAIN && (epi == EPI_SLOPE) != w_mn) return nullptr;
  switch (*row) {
    case 0: return kernel_of<DENSE, false, EPI_PLAIN>(pair);
    case 1: return kernel_of<DENSE, false, EPI_ACT>(pair);
    case 2: return kernel_of<DENSE, true, EPI_PLAIN>(pair);
    case 3: return kernel_of<DENSE, true, EPI_SLOPE>(pair);
    case 4: return kernel_of<ROWS, false, EPI_PLAIN>(pair);
    case 5: return kernel_of<ROWS, false, EPI_ACT>(pair);
    case 6: return kernel_of<ROWS, true, EPI_PLAIN>(pair);
    case 7: return kernel_of<ROWS, true, EPI_SLOPE>(pair);
  }
  return nullptr;
}

}  // namespace

namespace kbs {

bool ring_of(const Config& c, bool w_mn, int K, int groups, int rows, Ring* out) {
  const int ctas = c.pair ? 2 : 1, step = c.pair ? 32 : 16;
  const int w_cols = c.bn / ctas;
  const int tok_cta = c.pair ? c.tok / 2 : c.tok;
  if (w_cols < 8 || w_cols > LANES || c.bn % (w_mn ? 64 * ctas : 8 * ctas) != 0 || c.tok < step || c.tok > 256 || c.tok % step != 0 ||
      c.split < 1 || c.split > (c.pair ? 4 : 8) || c.split > ceil_div(K, BK) || (groups > 0 && c.split > 1)) {
    return false;
  }
  // Grouped rows: most blocks are shorter than `tok`.  Boxes of half the expected block fetch little in vain and a warp issues
  // two of them in the time the weights take (64 groups of 128 rows, 2048 x 1024: boxes of 32 rows 73.7 us, so 67.7).
  out->xbox = tok_cta;
  if (groups > 0) {
    const double n = static_cast<double>(rows) / groups, fits = n + 2.0 * sqrt(n);
    const int expect = fits < c.tok ? (static_cast<int>(fits) / step + 1) * step / ctas : tok_cta;
    out->xbox = ceil_div(expect, 16) * 8;
    if (out->xbox < 16) out->xbox = 16;
    if (out->xbox > tok_cta) out->xbox = tok_cta;
  }
  out->w_slot = w_cols * BK * 2;
  out->x_slot = ceil_div(tok_cta, out->xbox) * out->xbox * BK * 2;
  const int room = kbl::SMEM_MAX - 1024 - BAR_BYTES - (groups > 0 ? (3 * groups + 1) * 4 : 4);
  out->stages = room / (out->w_slot + out->x_slot);
  if (out->stages > MAX_STAGES) out->stages = MAX_STAGES;
  // The MMA reads 128 rows from the last slot of the weights on, of a narrower tile too: the token slots lie behind it.
  // The partial tiles of a split are exchanged through the ring.
  return out->stages >= 2 && out->stages * out->x_slot + out->w_slot >= LANES * BK * 2 &&
         (c.split == 1 || ceil_div(ceil_div(c.tok, CHUNK), c.split) * (c.split - 1) * LANES * CHUNK * 4 <= out->stages * (out->w_slot + out->x_slot));
}

int launch(const KbLocalGemmArgs& a, const Config& c, int dev, int cap, bool timing, void* stream) {
  const bool rows = a.kind == KB_LOCAL_ROWS, w_mn = a.b_mn != 0;
  const int ctas = c.pair ? 2 : 1;
  const int w_cols = c.bn / ctas;
  Ring ring;
  if (!ring_of(c, w_mn, a.K, rows ? a.groups : 0, a.expect > 0 ? a.expect : a.M, &ring)) {
    kb::set_error("kb_gemm_local: exchanged tile configuration pair=%d bn=%d tok=%d split=%d does not fit the problem", (int)c.pair, c.bn,
                  c.tok, c.split);
    return KB_ERR_ARG;
  }
  Params p;
  memset(&p, 0, sizeof(p));
  p.M = a.M;
  p.N = a.N;
  p.K = a.K;
  p.KB = ceil_div(a.K, BK);
  p.NB = ceil_div(a.N, c.bn);
  p.MB = ceil_div(a.M, c.tok);
  p.per = kbl::Div::by(rows ? p.NB : p.MB);
  p.bn = c.bn;
  p.tok = c.tok;
  p.groups = rows ? a.groups : 0;
  p.split = c.split;
  p.xbox = ring.xbox;
  p.w_slot = ring.w_slot;
  p.x_slot = ring.x_slot;
  p.stages = ring.stages;
  p.act = a.act;
  p.early = a.early != 0 ? 1 : 0;
  p.bias = static_cast<const bf16*>(a.bias);
  p.bias_scale = a.bias_scale;
  p.w = kbl::prefetches(a) ? static_cast<const bf16*>(a.B) : nullptr;
  p.out = static_cast<bf16*>(a.out);
  p.pre_out = static_cast<bf16*>(a.pre_out);
  p.pre_in = static_cast<const bf16*>(a.pre_in);
  p.row_start = a.row_start;
  p.row_count = a.row_count;
  p.status = a.status;
  p.limit_ns = a.wait_limit_ns ? a.wait_limit_ns : 2000000000ull;
  p.timing = timing ? 1 : 0;
  const uint64_t wz = rows ? a.groups : 1;
  int rc = kbl::make_tmap3(&p.tmX, a.A, a.K, a.M, 1, BK, p.xbox);
  if (rc != KB_OK) return rc;
  // [groups][N / 64][K][64]: the two blocks of 64 columns in one load; otherwise two loads, clipped at N
  p.w_whole = w_mn && a.N % 64 == 0 ? 1 : 0;
  rc = p.w_whole ? kbl::make_tmap4_blocks(&p.tmW, a.B, a.N, a.K, wz, BK, w_cols / 64)
       : w_mn ? kbl::make_tmap3(&p.tmW, a.B, a.N, a.K, wz, 64, BK) : kbl::make_tmap3(&p.tmW, a.B, a.K, a.N, wz, BK, w_cols);
  if (rc != KB_OK) return rc;

  const int cluster = ctas * c.split;
  const long long blocks = rows ? a.M / c.tok + static_cast<long long>(a.groups) : p.MB;  // rows: at most one partly filled block per group
  long long grid = blocks * p.NB * cluster;
  if (c.split == 1 && grid > cap / ctas * ctas) grid = cap / ctas * ctas;
  const int epi = a.pre_in != nullptr ? EPI_SLOPE : a.act != kbl::ACT_NONE ? EPI_ACT : EPI_PLAIN;
  int row = 0;
  const void* fn = find_kernel(a.kind, w_mn, epi, c.pair, &row);
  if (fn == nullptr) {
    kb::set_error("kb_gemm_local: no kernel for kind %d, weights along N %d, epilogue %d", a.kind, (int)w_mn, epi);
    return KB_ERR_UNSUPPORTED;
  }
  static bool attr_set[64][2][8] = {};
  if (dev < 0 || dev >= 64 || !attr_set[dev][c.pair][row]) {
    KB_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kbl::SMEM_MAX));
    if (dev >= 0 && dev < 64) attr_set[dev][c.pair][row] = true;
  }
  const bool overlapped = kbl::overlaps(cluster, c.split, static_cast<int>(grid), cap, 2.0 * a.N * a.K);
  return kbl::launch_clusters(fn, static_cast<int>(grid), THREADS, cluster, overlapped, &p, stream);
}

}  // namespace kbs
