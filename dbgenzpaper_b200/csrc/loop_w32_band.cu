// loop_w32_band.cu -- the warp-level FP32 loop for banded factors: the
// contraction over the band only, operands in three BF16 parts (FP32's 24
// bits), since the banded loop's FP32 modes multiply FP32 operands.
#include "loop_w32_impl.cuh"

#ifndef W32B_G
#define W32B_G 32
#define W32B_C 4
#endif

int dbgz_loop_w32_band(dbgz_problem *p, const PassArgs &pa, double *partials, int64_t n_tiles) {
  return w32_launch<3, W32B_G, W32B_C>(p, pa, partials, n_tiles, p->bandwidth);
}
