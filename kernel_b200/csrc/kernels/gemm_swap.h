// Products with exchanged operands (gemm_swap.cu), for the launcher of the single-GPU family (gemm_local.cu).
#pragma once
#include "../include/kb200.h"

namespace kbs {

struct Config {
  bool pair = false;
  int bn = 128;   // output columns of a tile
  int tok = 128;  // most token rows of a tile
  int split = 1;
};

// Shared memory of a configuration: rows of one box of X, bytes of a stage of the weights and of X, stages.
struct Ring {
  int xbox, w_slot, x_slot, stages;
};
// False where the kernel cannot run it: the choice of a tile skips such a configuration, the launcher refuses it.
// `groups`: 0 for a dense product; `rows`: rows expected in all groups together.
bool ring_of(const Config& c, bool w_mn, int K, int groups, int rows, Ring* out);

// Launches a dense or grouped-rows product whose arguments kb_gemm_local has checked.
int launch(const KbLocalGemmArgs& a, const Config& c, int dev, int cap, bool timing, void* stream);

}  // namespace kbs
