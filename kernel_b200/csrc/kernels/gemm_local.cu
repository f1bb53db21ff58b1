// Host side of the single-GPU tcgen05 GEMM family (device code: gemm_local.cuh).
#include "gemm_local.cuh"

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <mutex>

#include "gemm_local_host.h"
#include "gemm_swap.h"

namespace {

using namespace kbl;

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


struct Config {
  bool pair;
  int bn, split;
  bool tall = false;  // pair with 256 rows per CTA
  int rows = 128;     // ROWS, one CTA: rows of a tile
};

// Ring stages of a configuration and whether the partial tiles of a split fit the ring.
int ring_stages(int a_slot, int b_slot, int tables) {
  const int n = (SMEM_MAX - 1024 - BAR_BYTES - tables) / (a_slot + b_slot);
  return n > MAX_STAGES ? MAX_STAGES : n;
}
bool exchange_fits(int a_rows, bool pair, int bn, int split) {
  const int a_slot = a_rows * BK * 2, b_slot = (pair ? bn / 2 : bn) * BK * 2;
  const int slot_rows = pair ? 128 : ceil_div(a_rows, 32) * 32;
  return ceil_div(bn / CHUNK_COLS, split) * (split - 1) * slot_rows * CHUNK_COLS * 4 <= ring_stages(a_slot, b_slot, 4) * (a_slot + b_slot);
}

// Columns a tile may have: multiples of 32; an operand that is contiguous along N
// comes in boxes of 64 columns per CTA.
bool bn_ok(int bn, bool pair, bool b_mn) {
  const int per_cta = pair ? bn / 2 : bn;
  return b_mn ? per_cta % 64 == 0 : bn % 32 == 0;
}

// Clusters of 1 to 8 CTAs that are resident at a time ([0] unused).  Clusters do not
// cross a group of SMs that share a GPC, so large ones leave SMs idle (148 SMs: 74
// pairs, but 33 clusters of 4 and 15 of 8).
struct Capacity {
  int clusters[9];
};

// Operands in and results out at 6.5 TB/s behind the latency of a launch, ns.
double memory_time(int M, int N, int K) {
  return 2.0 * (static_cast<double>(M) * K + static_cast<double>(N) * K + static_cast<double>(M) * N) / 6500.0 + 6600.0;
}

// Picks the tile shape (one CTA, pair, 512-row pair), its columns and the split of K.
//
// Model of the kernel's time in ns, constants fitted to 190 shapes x all configurations
// on a B200 (M 2 to 16000, N and K 1000 to 29000; all three operand layouts; launches
// back to back in a graph): the picked configuration is 1.8 % slower than the best one
// on average.
//   k block   the tensor pipe needs 300 for 256 columns, tiles narrower than about 190
//             columns do not get faster (the operands of a single CTA's MMAs take
//             a third more shared-memory bandwidth); operand bytes arrive at 95 per ns
//             and SM, a little slower in the many small boxes of M/N-contiguous tensors
//   wave      2000 between the tiles of a CTA, the epilogue's last part is exposed
//             once, with 512-row tiles (no second accumulator) in every wave
//   split     one barrier more and the exchange of (split - 1) / split of a tile
//   memory    everything read and written once at 6.5 TB/s
// The configurations differ most where few tiles leave SMs idle (GPU time, launches back to back
// in a graph, three weights in turn; one CTA with 256 columns and no split against the pick):
// 64 x 7168 x 18432 88.5 and 45.1 us, 256 x 4096 x 14336 85.1 and 30.5, 2048 x 2880 x 2880 (in the
// L2) 35.1 and 24.4.  512-row tiles move 25 % fewer operand bytes
// per flop and win where K is long (8192 x 8192 x 29568: 3030 and 2840 us under the power cap).  An activation or a slope takes
// their epilogue longer in every wave, where a pair's runs under the next tile's products; pairs and 512-row tiles, us:
//                           plain        gelu, value kept     slope of gelu
//   8192 x 14336 x 4096    678   708        731   850           762   855
//   8192 x 29568 x 8192   2830  2858       2831  3163          3068  3113
// Not where K is an odd multiple of 8: rows along K then start inside a 32-byte sector, every 128 bytes of a box cost five
// sectors, and the operand bytes that 512-row tiles save are worth more.  Products that get such a tile without the 10 us (gelu, silu,
// relu; repeated), the picked tile above the better one on average without / with them; for the slope what replaces it against it:
//                   45 each: value dropped   kept            70 with a slope
//   K % 16 = 0               3.3  0.5 %      3.6   0.5 %     0.94
//   K % 16 = 8               0.0 10.2 %      0.0  11.0 %     1.04
// 8009 x 13128 x 8424 with gelu 1503 us, pairs 1852; 7974 x 21272 x 6984 with a slope 2423, exchanged pairs 2875.
Config choose_config(int M, int N, int K, bool a_mn, bool b_mn, const Capacity& cap, int shape, bool act, double* cost = nullptr) {
  Config best = {false, 256, 1};
  double best_t = 1e30, best_cost = 1e30;
  const int KB = ceil_div(K, BK);
  const double memory = memory_time(M, N, K);
  for (int s = 0; s < 3; ++s) {
    if (shape >= 0 ? s != shape : s != 0 && (M <= 128 || cap.clusters[2] < 1)) continue;
    const bool pair = s > 0, tall = s == 2;
    const int rows = tall ? 256 : (!pair && !a_mn && M < 128) ? ceil_div(M, 8) * 8 : 128;  // rows of A per stage
    for (int bn = 64; bn <= 256; bn += 32) {
      if (!bn_ok(bn, pair, b_mn) || (tall && bn != 256)) continue;
      const double tiles = static_cast<double>(ceil_div(M, 128 << s)) * ceil_div(N, bn);
      const double mma = 300.0 * (bn < 190 ? 190 : bn) / 256.0 * (tall ? 2.0 : pair ? 1.0 : 1.33);
      const double load = 128.0 * (rows + (pair ? bn / 2 : bn)) / 95.0 * (b_mn ? 1.07 : 1.0);
      const double k_block = mma > load ? mma : load;
      const double epilogue = 2000.0 * bn / 256.0 * (tall ? 2.0 : 1.0);
      for (int split = 1; split <= (tall ? 1 : pair ? 4 : 8); ++split) {
        const int units = cap.clusters[(pair ? 2 : 1) * split];
        if (split > 1 && (tiles > units || KB < 4 * split || !exchange_fits(rows, pair, bn, split))) continue;
        const double waves = units > 0 ? static_cast<double>((static_cast<long long>(tiles) + units - 1) / units) : 1e9;
        double t = 2000.0 + waves * (ceil_div(KB, split) * k_block + 2000.0) + epilogue + (pair ? 1000.0 : 0.0);
        if (tall) t += waves * (1.25 * epilogue + (act && K % 16 == 0 ? 10000.0 : 0.0));
        if (split > 1) t += 1300.0 + 2200.0 * bn / 256.0 * (split - 1) / split;
        // Launched behind the previous kernel instead of under its end.  Not so for the long reads that are launched in order
        // because that is faster (4 x 14488 x 16616, weights along N: 86.6 us split in two, 104 unsplit).
        const int ctas = (pair ? 2 : 1) * split;
        const bool late = ctas % 2 != 0 && !overlaps(ctas, split, static_cast<int>(tiles) * ctas, cap.clusters[1], 2.0 * N * K);
        const double in_order = late ? 1500.0 : 0.0;
        const double both = (t > memory ? t + 0.05 * memory : memory + 0.05 * t) + in_order;
        t = (t > memory ? t : memory) + in_order;
        if (t < best_t) {
          best_t = t;
          best_cost = both;
          best = {pair, bn, split, tall};
        }
      }
    }
  }
  if (cost != nullptr) *cost = best_cost;
  return best;
}

// A tenth of the tensor time, ns, of all rows and columns computed, padding included: under the power cap the energy of
// products of zeros and stale rows comes out of the clock.
double mma_energy(double rows, double cols, double K) { return 0.1 * 2.0 * rows * cols * K / 1.6e6; }

// Grouped rows.  The counts stay on the device, so the number of row blocks is an
// estimate from the average group: one if it fits a tile with two standard deviations
// to spare, else half a block of padding per group.  The rest is the model of the dense
// products.  With few rows the weights are the traffic and every shape that keeps the
// SMs loading is near the memory time; the second-order term breaks such ties.
//   64 experts, 2048 x 1024, 3 rows each: 32 x 256 tiles 45 us, 32 x 64 (first version) 68 us
// The epilogue that reads saved values back costs a pair more than one CTA (a pair's
// accumulators are free only when both have stored): pairs from about 400 rows per group on.
// Pair and one CTA in us, cold L2, equal groups (the line costs up to 10 % on its wrong sides, where N or K is
// long below it and at 640 rows above it):
//   rows per group            128         256         320         384         448         512         640
//   64 of [2048, 1024]     102  84    113 107    158 125    147 135    153 152    161 161    212 192
//   32 of [2048, 2048]     101  82    107 102    150 123    143 131    145 145    151 151    204 183
//   8 of [4096, 4096]       80  75     84  88    120 111    121 113    121 133    125 139    173 164
//   12 of [4096, 1536]      60  56     64  64     76  82     76  84     78  86     80  87     99 109
// Without that epilogue the model decides; its pairs cost 6 to 10 % at 128 rows per group of [2048, 1024] (76 and 69 us):
//   64 experts, 128 rows each: 128 x 192 tiles 61 us;  8 experts, 1000 rows of 4096 x 4096: pairs 198 us, one CTA 218 us
Config rows_plain_config(int M, int groups, int N, int K, bool b_mn, int sms, int shape, bool slope, double* cost_out) {
  Config best;
  best.bn = b_mn ? 128 : 256;
  best.pair = shape > 0;
  best.split = 1;
  double best_t = 1e30;
  const int KB = ceil_div(K, BK);
  const double n = static_cast<double>(M) / groups;
  const double used = n < 1.0 ? n : 1.0;  // share of groups that have rows
  const double memory = 2.0 * (used * groups * N * static_cast<double>(K) + static_cast<double>(M) * (N + K)) / 6500.0 + 6600.0;
  for (int s = 0; s < 4; ++s) {
    const bool pair = s == 3;
    if (shape >= 0 ? pair != (shape > 0) : pair && (sms < 2 || (slope && n < 448.0))) continue;
    const int rows = pair ? 256 : 32 << s;
    const double blocks = n + 2.0 * sqrt(n) <= rows ? used : n / rows + 0.5;
    for (int bn = 64; bn <= 256; bn += 64) {
      if (!bn_ok(bn, pair, b_mn)) continue;
      const double tiles = groups * blocks * ceil_div(N, bn);
      const double units = pair ? sms / 2 : sms;
      const double waves = tiles <= units ? 1.0 : tiles / units + 0.5;
      const double mma = 300.0 * (bn < 190 ? 190 : bn) / 256.0 * (pair ? 1.0 : 1.33);
      const double load = 128.0 * ((pair ? 128 : rows) + (pair ? bn / 2 : bn)) / 95.0 * (b_mn ? 1.07 : 1.0);
      const double t = 2000.0 + waves * (KB * (mma > load ? mma : load) + 2000.0) + 2000.0 * bn / 256.0 + (pair ? 1000.0 : 0.0);
      const double cost = t > memory ? t + 0.1 * memory : memory + 0.1 * t;
      if (cost < best_t) {
        best_t = cost;
        // the MMA computes 128 rows (256 for a pair) of every tile
        *cost_out = cost + mma_energy(groups * blocks * (pair ? 256.0 : 128.0), static_cast<double>(ceil_div(N, bn)) * bn, K);
        best.pair = pair;
        best.bn = bn;
        best.rows = pair ? 128 : rows;
      }
    }
  }
  return best;
}

// Time of a k block of a tile with exchanged operands, ns: constants as above; the issuing warps need `box` for each box of the
// tokens, however narrow the tile.
double swap_k_block(bool pair, int w_cols, int tok, bool w_mn, int boxes, double box) {
  const double mma = 300.0 * tok / 256.0 * (pair ? 1.0 : 1.33);
  const double load = 128.0 * (w_cols + (pair ? tok / 2 : tok)) / 95.0 * (w_mn ? 1.07 : 1.0);
  const double issue = boxes * box;
  const double t = mma > load ? mma : load;
  return t > issue ? t : issue;
}

// Dense product with exchanged operands: rows in blocks of at most 256, columns and split so that the tiles fill the chip.  The rows of
// a stage are one box, 170 ns in one CTA, 190 in a pair.  With the 130 of grouped rows' boxes, which a pair issues by twos, a quarter
// of the products of at most 64 rows gets another tile; repeated, of 60 of them (and of 50, weights along N) 25 (29) take more than 3 %
// longer, 8 (4) less:
//   1 x 23464 x 1504 14.7 us, pairs 16.4    7 x 9592 x 7560 31.0 and 34.3    weights along N: 23 x 25792 x 7536 67.8 and 77.9
double choose_swap(int M, int N, int K, bool w_mn, const Capacity& cap, int shape, kbs::Config* best) {
  double best_t = 1e30;
  const int KB = ceil_div(K, BK), mb = ceil_div(M, 256);
  const double memory = memory_time(M, N, K);
  for (int s = 0; s < 2; ++s) {
    const bool pair = s == 1;
    if (shape >= 3 ? s != shape - 3 : pair && cap.clusters[2] < 1) continue;
    const int step = pair ? 32 : 16;
    const int tok = ceil_div(ceil_div(M, mb), step) * step;
    for (int w_cols = w_mn ? 64 : 32; w_cols <= 128; w_cols += w_mn ? 64 : 8) {
      const int bn = pair ? 2 * w_cols : w_cols;
      const double tiles = static_cast<double>(mb) * ceil_div(N, bn);
      const double k_block = swap_k_block(pair, w_cols, tok, w_mn, 1, pair ? 190.0 : 170.0);
      for (int split = 1; split <= (pair ? 4 : 8); ++split) {
        const int ctas = (pair ? 2 : 1) * split;
        const int units = cap.clusters[ctas];
        if (split > 1 && (tiles > units || KB < 4 * split)) continue;
        kbs::Config c;
        c.pair = pair;
        c.bn = bn;
        c.tok = tok;
        c.split = split;
        kbs::Ring ring;
        if (!kbs::ring_of(c, w_mn, K, 0, M, &ring)) continue;
        const double waves = units > 0 ? static_cast<double>((static_cast<long long>(tiles) + units - 1) / units) : 1e9;
        double t = 2000.0 + waves * (ceil_div(KB, split) * k_block + 1500.0) + 2000.0 * tok / 256.0 + (pair ? 1000.0 : 0.0);
        if (split > 1) t += 800.0 + 2200.0 * tok / 256.0 * (split - 1) / split;
        t = t > memory ? t + 0.05 * memory : memory + 0.05 * t;
        if (split > 1 && !overlaps(ctas, split, static_cast<int>(tiles) * ctas, cap.clusters[1], 2.0 * N * K)) t += 1500.0;
        if (t < best_t) {
          best_t = t;
          *best = c;
        }
      }
    }
  }
  return best_t;
}

// Grouped rows with exchanged operands; the same estimates.  A box takes 170 ns, a pair's 130 where there are several, which go by twos,
// else 190 (16 groups of 0.2 rows, 832 x 3600: one CTA 14.3 us, pairs, which 130 would take, 16.4).
kbs::Config rows_swap_config(int M, int groups, int N, int K, bool w_mn, int sms, int shape, double* cost_out) {
  kbs::Config best;
  double best_t = 1e30;
  const int KB = ceil_div(K, BK);
  const double n = static_cast<double>(M) / groups;
  const double used = n < 1.0 ? n : 1.0;  // share of groups that have rows
  const double memory = 2.0 * (used * groups * N * static_cast<double>(K) + static_cast<double>(M) * (N + K)) / 6500.0 + 6600.0;
  for (int s = 0; s < 2; ++s) {
    const bool pair = s == 1;
    if (shape >= 0 ? s != shape - 3 : pair && sms < 2) continue;
    const int step = pair ? 32 : 16;
    for (int tok = 64; tok <= 256; tok *= 2) {
      const double fits = n + 2.0 * sqrt(n);
      const double blocks = fits <= tok ? used : n / tok + 0.5;
      const int cols = ceil_div(static_cast<int>(fits < tok ? fits : tok) + 1, step) * step;  // of a block
      for (int w_cols = 64; w_cols <= 128; w_cols += 64) {
        const int bn = pair ? 2 * w_cols : w_cols;
        kbs::Config c;
        c.pair = pair;
        c.bn = bn;
        c.tok = tok;
        kbs::Ring ring;
        if (!kbs::ring_of(c, w_mn, K, groups, M, &ring)) continue;
        const double tiles = groups * blocks * ceil_div(N, bn);
        const double units = pair ? sms / 2 : sms;
        const double waves = tiles <= units ? 1.0 : tiles / units + 0.5;
        // The tile is chosen as if the tokens came in one box, its cost counts the boxes: 8 groups of 121 rows of [640, 2960], in
        // pairs, take 15.9 us on the M side and 20.7 here.
        const int block = cols < tok ? cols : tok;
        const int boxes = ceil_div(block, (pair ? 2 : 1) * ring.xbox);
        auto cost_of = [&](int boxes_counted) {
          const double t = 2000.0 + waves * (KB * swap_k_block(pair, w_cols, block, w_mn, boxes_counted, !pair ? 170.0 : boxes > 1 ? 130.0 : 190.0) + 1000.0) + 2000.0 * cols / 256.0 + (pair ? 2000.0 : 0.0);
          return t > memory ? t + 0.1 * memory : memory + 0.1 * t;
        };
        const double cost = cost_of(1);
        if (cost < best_t) {
          best_t = cost;
          *cost_out = cost_of(boxes) +
                      mma_energy(groups * blocks * cols, static_cast<double>(ceil_div(N, bn)) * (pair ? 256.0 : 128.0), K);
          best = c;
        }
      }
    }
  }
  return best;
}

// Contractions over a group's rows.  About one k block: the outputs are all of the traffic, tiles of one CTA.  More: pairs, which
// fetch a third fewer operand bytes for the same output.  One CTA and pair in us, three outputs in turn, Poisson row counts:
//   rows per group           32          64          80          96         128         160         192         256
//   64 of 2048 x 1024      57  58      56  59      61  61      63  61      69  64      78  73      85  79     101  94
//   8 of 4096 x 4096       54  55      53  54      60  57      61  57      71  63      77  71      86  76     104  83
//   128 of 1024 x 768      45  46      46  50      49  49      50  50      61  52      64  55      70  64      83  73
//   32 of 2040 x 1000      35  37      40  36      42  39      44  39      48  43      53  46      58  50      67  57
// (Before the second CTA's epilogue gave its accumulator back without a fence, a pair took 93, 86, 76 and 53 at 128 rows.)
// Up to 224 rows that holds from three waves of pairs' tiles on, below six only if their taller tiles are no more than 1/16 padding.  One CTA
// and pair: 8 groups of 171 rows, 832 x 1088 7.1 9.0, of 69, 640 x 1024 6.1 7.1; 16 of 74, 896 x 1408 12.4 13.5.  79 products (66 to 223
// rows, 8 to 128 groups, M and N 512 to 4096): 0.4 % above the better tile on average and 2 more than 3 %; by the rows alone 2.4 % and 17.
Config contract_config(int M, int N, int rows, int groups, int sms, int shape) {
  Config c;
  c.bn = N <= 128 ? 128 : 256;
  const double wide = static_cast<double>(groups) * ceil_div(N, c.bn);
  const double ones = wide * ceil_div(M, 128), pairs = wide * ceil_div(M, 256), wave = sms / 2;
  const bool enough = pairs >= 6.0 * wave || (pairs >= 3.0 * wave && 32.0 * pairs <= 17.0 * ones);
  c.pair = shape >= 0 ? shape > 0 : M > 128 && (rows / groups >= 224 || (rows / groups >= 72 && enough));
  if (N <= 64 && !c.pair) c.bn = 64;
  c.split = 1;
  return c;
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

// Without a device to ask: what a B200 reports, scaled.
Capacity estimated_capacity(int sms) {
  static const int on_148[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  Capacity c;
  for (int i = 0; i < 9; ++i) c.clusters[i] = on_148[i] * sms / 148;
  return c;
}

template <Kind kKind, bool kAMn, bool kBMn, Epi kEpi>
const void* kernel_of(const Config& c) {
  if constexpr (kKind == DENSE) {
    if (c.tall) return (const void*)gemm_local_kernel<kKind, true, kAMn, kBMn, 2, kEpi>;
  }
  return c.pair ? (const void*)gemm_local_kernel<kKind, true, kAMn, kBMn, 1, kEpi>
                : (const void*)gemm_local_kernel<kKind, false, kAMn, kBMn, 1, kEpi>;
}

// The kernels that exist: an activation follows a product whose weights are
// contiguous along K (forward), a slope one whose weights are contiguous along N
// (backward); row 3 * variant + epilogue of the attribute cache.
const void* find_kernel(int kind, bool a_mn, bool b_mn, int epi, const Config& c, int* row) {
  const int variant = kind == ROWS ? (b_mn ? 4 : 3) : kind == CONTRACT ? 5 : a_mn ? 2 : b_mn ? 1 : 0;
  *row = 3 * variant + epi;
  switch (*row) {
    case 0: return kernel_of<DENSE, false, false, EPI_PLAIN>(c);
    case 1: return kernel_of<DENSE, false, false, EPI_ACT>(c);
    case 3: return kernel_of<DENSE, false, true, EPI_PLAIN>(c);
    case 5: return kernel_of<DENSE, false, true, EPI_SLOPE>(c);
    case 6: return kernel_of<DENSE, true, true, EPI_PLAIN>(c);
    case 9: return kernel_of<ROWS, false, false, EPI_PLAIN>(c);
    case 10: return kernel_of<ROWS, false, false, EPI_ACT>(c);
    case 12: return kernel_of<ROWS, false, true, EPI_PLAIN>(c);
    case 14: return kernel_of<ROWS, false, true, EPI_SLOPE>(c);
    case 15: return kernel_of<CONTRACT, true, true, EPI_PLAIN>(c);
  }
  return nullptr;
}

}  // namespace

namespace {

// Asked once per device.
int device_capacity(int dev, int sms, Capacity* out) {
  static Capacity cached_clusters[64];
  static std::atomic<int> known[64];
  const bool keep = dev >= 0 && dev < 64;
  if (keep && known[dev].load(std::memory_order_acquire)) {
    *out = cached_clusters[dev];
    return KB_OK;
  }
  Capacity c = {{0, sms}};
  const void* fn = (const void*)gemm_local_kernel<DENSE, false, false, false, 1, EPI_PLAIN>;
  KB_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
  for (int size = 2; size <= 8; ++size) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(size * sms);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_MAX;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    KB_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, fn, &cfg));
    c.clusters[size] = n;
  }
  if (keep) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (!known[dev].load(std::memory_order_relaxed)) {
      cached_clusters[dev] = c;
      known[dev].store(1, std::memory_order_release);
    }
  }
  *out = c;
  return KB_OK;
}

// The choice depends on the sizes alone and a program calls with the same ones again
// and again: a small table per thread, dense and grouped products together, remembers it (a search takes 0.3 to 1.7 us).
struct Choice {
  bool swap;      // exchanged operands
  Config c;
  kbs::Config s;
};
struct Remembered {
  int M, N, K, groups, key, dev;
  Choice c;
};
Remembered& remembered(int M, int N, int K, int groups, int key) {
  thread_local Remembered table[64] = {};
  const uint32_t h = (static_cast<uint32_t>(M) * 0x9e3779b1u) ^ (static_cast<uint32_t>(N) * 0x85ebca6bu) ^
                     (static_cast<uint32_t>(K) * 0xc2b2ae35u) ^ static_cast<uint32_t>(key + groups);
  return table[(h ^ (h >> 15)) & 63u];
}
// What the exchanged kernel gains, ns, by fetching weights under the end of the previous launch, which the other one does not
// do.  500 MLPs (1 to 1200 tokens) and 582 MoE layers: with 0, 1500 and 3000 a pair of products takes 0.856, 0.852 and 0.854 of what it
// took on the M side in order (MLP), 0.919, 0.906 and 0.905 (MoE); 4, none and 2 MLPs take more than 3 % longer, 10, 24 and 32 layers.
constexpr double EARLY = 1500.0;

// Rows on the tensor cores' M side or on their N side: what the two models say, plus the energy, plus what 2330 products (1 to
// 8192 rows, all layouts and epilogues, three weights in turn) showed them to leave out: a split costs more than they say,
// more so with many tokens, whose partial tiles are exchanged; tiles that are not split fall a little further short of the
// memory's rate, exchanged ones of more than 128 rows too.  Constants fitted between 330 near ties repeated for 0.1 s each, at the
// power cap, where the energy counts for most, and 2000 short bursts.  The picked kind takes 1.2 % and 1.6 % more than the better
// one on average (always the M side 5.0 and 5.5 %, always exchanged 3.9 and 5.0 %).  Near ties keep the rows on the M side, whose
// epilogue stores wider vectors, except with a slope, whose saved values it reads back with a row per lane.  Bursts, us, M side and
// exchanged, the picked one marked:
//   1 x 8192 x 8192   27.2  26.4*   40 x 2840 x 1392    7.8   7.2*   64 x 7168 x 18432   47.2  48.1*   100 x 4096 x 14336   27.9* 28.3
//   165 x 2920 x 1080 10.4* 12.0    200 x 8192 x 8192  33.8* 33.4    300 x 1024 x 1024    9.2*  9.9    330 x 6296 x 1304    14.0* 13.8
//   400 x 25000 x 1504 35.1 31.2*   90 x 1104 x 20000  16.4  17.0*   195 x 26136 x 3200  38.9* 42.0    256 x 4096 x 14336   36.5* 46.0
Choice choose(int M, int N, int K, bool a_mn, bool b_mn, const Capacity& cap, int shape, bool act, bool slope, bool early) {
  Choice r = {};
  double plain = 0.0;
  if (shape < 3) r.c = choose_config(M, N, K, a_mn, b_mn, cap, shape, act, &plain);
  if (a_mn || (shape >= 0 && shape < 3)) return r;
  const double other = choose_swap(M, N, K, b_mn, cap, shape, &r.s);
  if (shape >= 3) {
    r.swap = true;
    return r;
  }
  const int tall = r.c.tall ? 512 : r.c.pair ? 256 : 128;
  const int lanes = r.s.pair ? 256 : 128;
  const double memory = memory_time(M, N, K);
  const double exchange = 3700.0 * r.s.tok / 256.0 * (r.s.split - 1) / r.s.split;
  const double cost_m = plain + 3.5 * mma_energy(static_cast<double>(ceil_div(M, tall)) * tall, static_cast<double>(ceil_div(N, r.c.bn)) * r.c.bn, K) +
                        (r.c.split > 1 ? 3000.0 : 0.167 * memory);
  const double cost_n = other + 3.5 * mma_energy(static_cast<double>(ceil_div(M, r.s.tok)) * r.s.tok, static_cast<double>(ceil_div(N, r.s.bn)) * lanes, K) +
                        (r.s.split > 1 ? 2300.0 + exchange : 0.174 * memory) + (M > 128 ? 0.12 * memory : 0.0);
  r.swap = cost_n - (early ? EARLY : 0.0) < (slope ? 1.05 : 0.97) * cost_m;
  return r;
}
int pick_config(int dev, int sms, int cap, int M, int N, int K, bool a_mn, bool b_mn, int shape, bool act, bool slope, bool early, Choice* out) {
  const int key = (a_mn ? 1 : 0) | (b_mn ? 2 : 0) | (act ? 1 << 27 : 0) | (slope ? 1 << 29 : 0) | (early ? 1 << 28 : 0) | ((shape + 1) << 2) | (cap << 5) | (1 << 30);
  Remembered& e = remembered(M, N, K, 0, key);
  if (e.M != M || e.N != N || e.K != K || e.groups != 0 || e.key != key || e.dev != dev) {
    Capacity have = estimated_capacity(sms);
    const int rc = dev < 0 ? KB_OK : device_capacity(dev, sms, &have);
    if (rc != KB_OK) return rc;
    for (int i = 1; i < 9; ++i) have.clusters[i] = have.clusters[i] * i <= cap ? have.clusters[i] : cap / i;
    e = {M, N, K, 0, key, dev, choose(M, N, K, a_mn, b_mn, have, shape, act, slope, early)};
  }
  *out = e.c;
  return KB_OK;
}
// Grouped rows; `rows` of them are expected.
Choice pick_rows(int cap, int rows, int groups, int N, int K, bool w_mn, int shape, bool slope, bool early) {
  const int key = (slope ? 1 : 0) | (early ? 1 << 28 : 0) | (w_mn ? 2 : 0) | ((shape + 1) << 2) | (cap << 5) | (1 << 30);
  Remembered& e = remembered(rows, N, K, groups, key);
  if (e.M != rows || e.N != N || e.K != K || e.groups != groups || e.key != key) {
    Choice r = {};
    double plain = 1e30, other = 1e30;
    if (shape < 3) r.c = rows_plain_config(rows, groups, N, K, w_mn, cap, shape, slope, &plain);
    if (shape < 0 || shape >= 3) r.s = rows_swap_config(rows, groups, N, K, w_mn, cap, shape, &other);
    // Groups of some blocks: little padding either way.  A slope favours the N side: the M side's epilogue reads the saved values
    // back with a row per lane and keeps the accumulator of a tile longer.  us, rows on the M side / exchanged:
    //   rows per group, [N, K]        3, [1024, 2048]   3, [760, 2728]   128, [1024, 2048]   250, [4096, 4096]   717, [544, 3008]
    //   forward with activation          47.6  45.5        99.5  89.4       75.3  67.7          98.5 101           25.3  26.7
    //   slope                            56.6  56.0         145   144       90.8  75.4           116  94.4         36.5  31.5
    // Limits, the time per box and a pair's 2000 ns fitted to 560 products in bursts (8 to 128 groups of 1 to 900 rows, Poisson
    // counts, N and K 512 to 4096), after boxes came by twos and pairs handed their accumulators on without a fence: forward
    // with activation, plain and slope take 1.4, 1.6 and 2.0 % more than the best tile of both kinds on average (before the fit 5.7, 3.6
    // and 3.0; always exchanged 1.3, 1.9 and 1.4, always the M side 9.5, 4.5 and 17), 84 of 558 more than 3 % (179).  That was with 1.25 below 32
    // rows and 130 ns for a pair's single box; 563 others of 0.1 to 31 rows take 1.4 % more than the best kind so, 1.8 with those.
    // 2316 products of 0.2 to 1200 rows per group, in order of the three: 3.1, 4.2 and 3.3 % above the fastest of one CTA and pair of
    // either kind (the fastest of five noisy times); kernels and rule before the fit took 9.7, 8.8 and 7.7 % more.
    const double limit = slope ? 1.14 : rows >= 192ll * groups ? 1.02 : rows >= 32ll * groups ? 0.99 : 1.05;
    r.swap = other - (early ? EARLY : 0.0) < limit * plain;
    e = {rows, N, K, groups, key, 0, r};
  }
  return e.c;
}

}  // namespace

extern "C" int kb_gemm_local_config(int M, int N, int K, int a_mn, int b_mn, int sms, int* pair, int* bn, int* split) {
  if (M <= 0 || N <= 0 || K <= 0 || sms < 2 || !pair || !bn || !split) return KB_ERR_ARG;
  const Config c = choose_config(M, N, K, a_mn != 0, b_mn != 0, estimated_capacity(sms), -1, false);
  *pair = c.tall ? 2 : c.pair ? 1 : 0;
  *bn = c.bn;
  *split = c.split;
  return KB_OK;
}

namespace {

struct Layout {
  bool contract, grouped, a_mn, b_mn;
};

// What does not depend on pointers or on a device.
int check_problem(const KbLocalGemmArgs* a, Layout* l) {
  if (a == nullptr) return KB_ERR_ARG;
  l->contract = a->kind == KB_LOCAL_CONTRACT;
  if (a->kind < 0 || a->kind > 2 || a->act < 0 || a->act > 3) {
    kb::set_error("kb_gemm_local: unknown kind %d or activation %d", a->kind, a->act);
    return KB_ERR_ARG;
  }
  l->a_mn = l->contract || a->a_mn;
  l->b_mn = l->contract || a->b_mn;
  l->grouped = a->kind != KB_LOCAL_DENSE;
  const bool a_mn = l->a_mn, b_mn = l->b_mn;
  // TMA rows are multiples of 16 bytes: the contiguous extent of every tensor is a multiple of 8.
  if (a->M <= 0 || a->N <= 0 || a->K <= 0 || a->N % 8 != 0 || (!a_mn && a->K % 8 != 0) || (!b_mn && a->K % 8 != 0) ||
      (a_mn && a->M % 8 != 0)) {
    kb::set_error("kb_gemm_local: need M,N,K > 0 and contiguous extents that are multiples of 8 (got %d %d %d)", a->M, a->N, a->K);
    return KB_ERR_ARG;
  }
  if (l->grouped && (a->groups < 1 || a->groups > MAX_GROUPS || a->row_start == nullptr || a->row_count == nullptr || a->bias != nullptr ||
                  (a->kind == KB_LOCAL_ROWS && a_mn))) {
    kb::set_error("kb_gemm_local: bad groups (%d, at most %d, with row tables, without bias)", a->groups, MAX_GROUPS);
    return KB_ERR_ARG;
  }
  if (a->kind == KB_LOCAL_DENSE && a_mn && !b_mn) {
    kb::set_error("kb_gemm_local: A contiguous along M is built only with B contiguous along N");
    return KB_ERR_UNSUPPORTED;
  }
  if ((a->pre_in != nullptr || a->pre_out != nullptr) && a->act == KB_ACT_NONE) {
    kb::set_error("kb_gemm_local: pre_in and pre_out belong to an activation");
    return KB_ERR_ARG;
  }
  return KB_OK;
}

// The tile a product gets: what is asked for, else what the sizes call for.
int pick_tile(const KbLocalGemmArgs* a, const Layout& l, int dev, int sms, int cap, Choice* out) {
  const int groups = l.grouped ? a->groups : 1;
  const int expect = a->expect > 0 ? a->expect : a->kind == KB_LOCAL_ROWS ? a->M : a->K;
  int shape = a->pair;  // -1: choose, 0: one CTA, 1: pair, 2: tall pair, 3 and 4: exchanged operands
  if (cap < 2 || env().no_pair) shape = shape >= 3 ? 3 : 0;
  Choice pick = {};
  if (a->kind == KB_LOCAL_ROWS) {
    pick = pick_rows(cap, expect, groups, a->N, a->K, l.b_mn, shape, a->pre_in != nullptr, a->early != 0);
  } else if (a->kind == KB_LOCAL_DENSE) {
    if (shape == 1 && a->M <= 128) shape = 0;  // a pair's second CTA would hold padding only
    const int rc = pick_config(dev, sms, cap, a->M, a->N, a->K, l.a_mn, l.b_mn, shape, a->act != ACT_NONE, a->pre_in != nullptr, a->early != 0, &pick);
    if (rc != KB_OK) return rc;
  } else {
    pick.c = contract_config(a->M, a->N, expect, groups, cap, shape);
  }
  if (shape < 3 && (a->bn > 0 || a->split > 0)) pick.swap = false;  // a tile of the other kind is asked for
  int* bn = pick.swap ? &pick.s.bn : &pick.c.bn;
  int* split = pick.swap ? &pick.s.split : &pick.c.split;
  if (a->bn > 0) *bn = a->bn;
  if (a->split > 0) *split = a->split;
  if (a->tok > 0) pick.s.tok = a->tok;
  *out = pick;
  return KB_OK;
}

// Contractions of groups that have about one k block.
bool one_k_block(const KbLocalGemmArgs* a) { return (a->expect > 0 ? a->expect : a->K) <= 56ll * a->groups; }

// Two stages of the ring instead of three: such a contraction waits for its stores, and loads that run ahead of them hold them up
// where the output does not fit the L2 and its rows start inside a 32-byte sector, fill whole lines or are few and long.  us, three
// stages and two:
//   64 groups of 22 rows, 3448 x 960   92.2  81.4    64 of 19, 3656 x 648   95.9  77.6    64 of 16, 2048 x 1024   56.1  51.5
//   64 of 24, 2504 x 1432             143.5 118.9    32 of 22, 2064 x 2888 110.4  93.4    128 of 6, 656 x 2160    85.3  80.2
// Elsewhere three: 32 of 24, 3792 x 1424 (rows of whole sectors) 63.9 and 72.1, 32 of 30, 2816 x 2848 94.2 and 103; 16 of 14,
// 792 x 1864 (47 MB) 15.0 and 15.6.  122 products of 4 to 56 rows per group take 0.2 % more than with the better number on average;
// always three 2.3 %, always two 4.4 %.
bool two_stages(const KbLocalGemmArgs* a, const Config& c) {
  return one_k_block(a) && !c.pair && c.bn == 256 && 2.0 * a->groups * a->M * a->N > 180e6 &&
         (a->N % 16 != 0 || a->N % 64 == 0 || a->N > 2 * a->M);
}

// Shared memory of a tile with the rows on the M side; false where the kernel cannot run it.
struct Ring {
  int a_rows, a_slot, b_slot, stages;
  int slot_rows;  // of an exchange slot of a split
};
bool ring_of(const KbLocalGemmArgs* a, const Layout& l, const Config& c, Ring* r) {
  if (c.bn < 32 || c.bn > 256 || !bn_ok(c.bn, c.pair, l.b_mn) || c.split < 1 || c.split > (c.pair ? 4 : 8) || c.split > ceil_div(a->K, BK) ||
      ((l.grouped || c.tall) && c.split > 1)) {
    return false;
  }
  // A single CTA whose rows are few brings in only those: the MMA reads 128 rows of
  // shared memory, what lies behind the box only reaches accumulator rows that are not
  // stored.
  r->a_rows = c.tall ? 256 : 128;
  if (a->kind == KB_LOCAL_ROWS && !c.pair) {
    r->a_rows = c.rows;
  } else if (!c.pair && !l.a_mn && a->M < 128) {
    r->a_rows = ceil_div(a->M, 8) * 8;
  }
  r->a_slot = r->a_rows * BK * 2;
  r->b_slot = (c.pair ? c.bn / 2 : c.bn) * BK * 2;
  const int tables = (l.grouped ? (3 * a->groups + 1) * 4 : 4) + (l.contract ? OUT_BYTES : 0);  // what the ring leaves room for
  r->stages = ring_stages(r->a_slot, r->b_slot, tables);
  if (l.contract && r->stages > 2 && two_stages(a, c)) r->stages = 2;
  r->slot_rows = c.pair ? 128 : ceil_div(r->a_rows, 32) * 32;
  // the last A slot is read up to 128 rows far: the B slots behind it cover that
  return r->stages >= 2 && r->stages * r->b_slot >= 16384 && (c.split == 1 || exchange_fits(r->a_rows, c.pair, c.bn, c.split));
}

}  // namespace

extern "C" int kb_gemm_local_pick(const KbLocalGemmArgs* a, int sms, KbLocalPick* out) {
  if (a == nullptr || out == nullptr || sms < 1) return KB_ERR_ARG;
  Layout l;
  Choice pick;
  int rc = check_problem(a, &l);
  const int cap = a->num_ctas > 0 && a->num_ctas < sms ? a->num_ctas : sms;
  if (rc == KB_OK) rc = pick_tile(a, l, -1, sms, cap, &pick);
  if (rc != KB_OK) return rc;
  const Config& c = pick.c;
  const kbs::Config& s = pick.s;
  if (pick.swap) *out = {1, s.pair, s.bn, s.tok, s.split};
  else *out = {0, c.tall ? 2 : c.pair, c.bn, c.tall ? 512 : c.pair ? 256 : a->kind == KB_LOCAL_ROWS ? c.rows : 128, c.split};
  const int cluster = (out->pair ? 2 : 1) * out->split;
  out->overlapped = overlaps(cluster, out->split, ceil_div(a->M, out->rows) * ceil_div(a->N, out->bn) * cluster, cap, 2.0 * a->N * a->K);
  out->ahead = prefetches(*a);
  Ring ring;
  kbs::Ring swap_ring;
  const int expect = a->expect > 0 ? a->expect : a->M;
  const bool fits = pick.swap ? kbs::ring_of(s, l.b_mn, a->K, l.grouped ? a->groups : 0, expect, &swap_ring) : ring_of(a, l, c, &ring);
  out->stages = !fits ? 0 : pick.swap ? swap_ring.stages : ring.stages;
  return fits ? KB_OK : KB_ERR_UNSUPPORTED;
}

extern "C" int kb_gemm_local(const KbLocalGemmArgs* a, void* stream_v) {
  Layout l;
  int rc = check_problem(a, &l);
  if (rc != KB_OK) return rc;
  const bool contract = l.contract, grouped = l.grouped, a_mn = l.a_mn, b_mn = l.b_mn;
  auto misaligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
  if (a->A == nullptr || a->B == nullptr || a->out == nullptr || misaligned(a->A) || misaligned(a->B) || misaligned(a->out) ||
      misaligned(a->bias) || misaligned(a->pre_out) || misaligned(a->pre_in)) {
    kb::set_error("kb_gemm_local: operand pointers must be given and 16-byte aligned");
    return KB_ERR_ARG;
  }
  int dev = 0, sms = 0;
  rc = device_info(&dev, &sms);
  if (rc != KB_OK) return rc;
  const int cap = a->num_ctas > 0 && a->num_ctas < sms ? a->num_ctas : sms;

  Choice pick;
  rc = pick_tile(a, l, dev, sms, cap, &pick);
  if (rc != KB_OK) return rc;
  if (pick.swap) return kbs::launch(*a, pick.s, dev, cap, env().timing, stream_v);
  const Config c = pick.c;
  const int groups = grouped ? a->groups : 1;
  Ring ring;
  if (!ring_of(a, l, c, &ring)) {
    kb::set_error("kb_gemm_local: tile configuration pair=%d bn=%d split=%d does not fit the problem", c.pair, c.bn, c.split);
    return KB_ERR_ARG;
  }

  Params p;
  memset(&p, 0, sizeof(p));
  p.M = a->M;
  p.N = a->N;
  p.K = a->K;
  p.a_rows = ring.a_rows;
  const int tile_rows = c.tall ? 512 : c.pair ? 256 : a->kind == KB_LOCAL_ROWS ? p.a_rows : 128;
  p.MBQ = ceil_div(a->M, tile_rows);
  p.NB = ceil_div(a->N, c.bn);
  p.KB = ceil_div(a->K, BK);
  p.bn = c.bn;
  p.group = (c.tall ? 4096 : 2048) / tile_rows;
  p.groups = grouped ? groups : 0;
  p.per = Div::by(contract ? p.MBQ * p.NB : grouped ? p.NB : p.group * p.NB);
  p.first = Div::by(contract ? p.MBQ : p.group);
  p.last = Div::by(p.MBQ % p.group);
  p.split = c.split;
  p.a_slot = ring.a_slot;
  p.b_slot = ring.b_slot;
  p.stages = ring.stages;
  p.slot_rows = ring.slot_rows;
  const int epi = a->pre_in != nullptr ? EPI_SLOPE : a->act != ACT_NONE ? EPI_ACT : EPI_PLAIN;
  auto wide = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31u) == 0; };
  p.wide = a->N % 16 == 0 && wide(a->out) && wide(a->pre_out) && wide(a->pre_in) ? 1 : 0;
  p.act = a->act;
  p.bias = static_cast<const bf16*>(a->bias);
  p.bias_scale = a->bias_scale;
  p.w = prefetches(*a) ? static_cast<const bf16*>(a->B) : nullptr;
  p.out = static_cast<bf16*>(a->out);
  p.pre_out = static_cast<bf16*>(a->pre_out);
  p.pre_in = static_cast<const bf16*>(a->pre_in);
  p.row_start = a->row_start;
  p.row_count = a->row_count;
  p.status = a->status;
  p.limit_ns = a->wait_limit_ns ? a->wait_limit_ns : 2000000000ull;
  p.timing = env().timing ? 1 : 0;

  const uint64_t bz = a->kind == KB_LOCAL_ROWS ? groups : 1;
  // A contraction over one k block waits for its stores, not for loads, and large boxes hold the stores up: 128 groups of 16 rows,
  // 512 x 2048, 58 us with a load per 64 columns, 61 with one per operand.
  const bool whole = !contract || !one_k_block(a);
  p.a_whole = whole && a_mn && a->M % 64 == 0 ? 1 : 0;
  p.b_whole = whole && b_mn && a->N % 64 == 0 ? 1 : 0;
  const int b_cols = c.pair ? c.bn / 2 : c.bn;
  rc = p.a_whole ? make_tmap4_blocks(&p.tmA, a->A, a->M, a->K, 1, BK, p.a_rows / 64)
       : a_mn ? make_tmap3(&p.tmA, a->A, a->M, a->K, 1, 64, BK) : make_tmap3(&p.tmA, a->A, a->K, a->M, 1, BK, p.a_rows);
  if (rc != KB_OK) return rc;
  rc = p.b_whole ? make_tmap4_blocks(&p.tmB, a->B, a->N, a->K, bz, BK, b_cols / 64)
       : b_mn ? make_tmap3(&p.tmB, a->B, a->N, a->K, bz, 64, BK) : make_tmap3(&p.tmB, a->B, a->K, a->N, bz, BK, b_cols);
  if (rc != KB_OK) return rc;
  if (contract) {
    rc = make_tmap3(&p.tmOut, a->out, a->N, a->M, groups, 64, 32);
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

  int kernel_row = 0;
  const void* fn = find_kernel(a->kind, a_mn, b_mn, epi, c, &kernel_row);
  if (fn == nullptr) {
    kb::set_error("kb_gemm_local: no kernel for kind %d, layouts %d %d, epilogue %d", a->kind, (int)a_mn, (int)b_mn, epi);
    return KB_ERR_UNSUPPORTED;
  }
  const int shape_row = c.tall ? 2 : c.pair ? 1 : 0;
  static bool attr_set[64][3][18] = {};
  if (dev < 0 || dev >= 64 || !attr_set[dev][shape_row][kernel_row]) {
    KB_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    if (dev >= 0 && dev < 64) attr_set[dev][shape_row][kernel_row] = true;
  }
  return launch_clusters(fn, grid, THREADS, cluster, overlaps(cluster, c.split, grid, cap, 2.0 * a->N * a->K), &p, stream_v);
}
