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

// Launches a dense or grouped-rows product whose arguments kb_gemm_local has checked.
int launch(const KbLocalGemmArgs& a, const Config& c, int dev, int cap, bool timing, void* stream);

}  // namespace kbs
