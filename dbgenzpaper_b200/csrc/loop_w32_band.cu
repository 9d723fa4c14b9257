// loop_w32_band.cu -- the warp-level FP32 loop for banded factors: the
// contraction over the band only, the products with earlier groups' y's on
// three BF16 parts (FP32's 24 bits), since the banded loop's FP32 modes multiply
// FP32 operands (rms error of the shifts' means at d = 600, bandwidths 5 to 100:
// 4.0e-7 to 7.8e-7, by the CSC loop's FP32 FMAs 5.5e-7 to 11.8e-7).
#include "loop_w32_impl.cuh"

int dbgz_loop_w32_band(dbgz_problem *p, const PassArgs &pa, double *partials, int64_t n_tiles) {
  return w32_launch<3, 32, 4>(p, pa, partials, n_tiles, p->bandwidth);
}
