// loop_w32_band.cu -- the warp-level FP32 loop for banded factors: the
// contraction over the band only, operands in three BF16 parts (FP32's 24
// bits), since the banded loop's FP32 modes multiply FP32 operands.
#include "loop_w32_impl.cuh"

int dbgz_loop_w32_band(dbgz_problem *p, const PassArgs &pa, double *partials, int64_t n_tiles) {
  return w32_launch<3, 32, 4>(p, pa, partials, n_tiles, p->bandwidth);
}
