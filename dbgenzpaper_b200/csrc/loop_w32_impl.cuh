// loop_w32_impl.cuh -- operand preparation and launch of the warp-level FP32
// loop (loop_w32_kernels.cuh) for one number of BF16 parts; loop_w32.cu and
// loop_w32_band.cu instantiate it (two files, compiled side by side).
#pragma once
#include <algorithm>

#include "loop_w32_kernels.cuh"

namespace {

// U^T panels in NPART BF16 parts (rows t = 1 .. d - 1 of ld entries from the
// first y-index that reaches the row's group) and the groups' FP32 coefficients.
template <int NPART, int G>
__global__ void k_w32_panels(const double *U, int64_t d, int64_t ld, int64_t band, uint16_t *u0, uint16_t *u1,
                             uint16_t *u2) {
  const int64_t t = blockIdx.y + (int64_t)gridDim.y * blockIdx.z + 1;
  if (t >= d) return;
  const int64_t g0 = (t - 1) / G * G, lofs = band > 0 ? w32::first_k<G>(g0, band) : 0;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < ld; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t l = lofs + j;
    double u = l < t ? U[t * d + l] : 0.0;
    uint16_t *o[3] = {u0, u1, u2};
#pragma unroll
    for (int p = 0; p < NPART; ++p) {
      const __nv_bfloat16 h = __double2bfloat16(u);
      o[p][t * ld + j] = __bfloat16_as_ushort(h);
      u -= (double)__bfloat162float(h);
    }
  }
}
__global__ void k_w32_tri(const double *U, int64_t d, int64_t n, float *tri) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= n) return;
  tri[e] = w32::tri_value(U, d, e);
}

template <int NPART, int G>
struct W32Layout {
  int64_t ld, rows_bytes, tri_n, ring_chunks, slot;
  W32Layout(int64_t d, int64_t band) {
    const int64_t nY = d - 1;
    ld = band > 0 ? (band + 15) / 16 * 16 + 16 + G : (nY + 63) / 64 * 64;
    rows_bytes = (d * ld * 2 + 255) / 256 * 256;
    tri_n = (nY + w32::SB - 1) / w32::SB * w32::kTri;
    ring_chunks = ld / w32::CH;
    slot = ring_chunks * 4 * NPART * 512;
  }
};

template <int NPART, int G>
int w32_operands(dbgz_problem *p, bool adj, int64_t band, DevBuf &b) {
  dbgz_ctx *ctx = p->ctx;
  const int64_t d = p->d;
  const W32Layout<NPART, G> L(d, band);
  if (b.p) return DBGZ_OK;
  if (adj && !p->Ub.p) DBGZ_TRY(dbgz_make_Ub(p));
  DBGZ_TRY(dbgz_ensure(ctx, b, (size_t)L.rows_bytes * NPART + sizeof(float) * (size_t)L.tri_n));
  const double *U = (const double *)(adj ? p->Ub.p : p->U.p);
  char *base = (char *)b.p;
  uint16_t *u[3];
  for (int i = 0; i < 3; ++i) u[i] = (uint16_t *)(base + (i < NPART ? i : 0) * L.rows_bytes);
  const unsigned gy = (unsigned)std::min<int64_t>(d - 1, 32768);
  k_w32_panels<NPART, G><<<dim3((unsigned)std::min<int64_t>((L.ld + 127) / 128, 4), gy, (unsigned)((d - 2 + gy) / gy)),
                           128, 0, ctx->stream>>>(U, d, L.ld, band, u[0], u[1], u[2]);
  dbgz_count_launch(ctx);
  k_w32_tri<<<(unsigned)((L.tri_n + 255) / 256), 256, 0, ctx->stream>>>(U, d, L.tri_n,
                                                                         (float *)(base + L.rows_bytes * NPART));
  dbgz_count_launch(ctx);
  DBGZ_CUDA_TRY(ctx, cudaGetLastError());
  return DBGZ_OK;
}

template <int NPART, int G, int CTAS, int GEN>
auto w32_pick(int kind, bool lower_inf) -> void (*)(w32::Params) {
  using namespace w32;
  // three parts with the stored state or the adjoint's spill at four CTAs an
  // SM: gradient of the d = 4000, bandwidth 64 problem 11.7 ms, 10.2 with three
  constexpr int CG = NPART > 2 ? CTAS - 1 : CTAS;
  switch (kind) {
    case kLoopForwardStore:
      if (lower_inf) return k_genz_w32<NPART, G, CG, pol::Forward<float, GEN, true, dbgz::StepFp32LowerInf>>;
      return k_genz_w32<NPART, G, CG, pol::Forward<float, GEN, true>>;
    case kLoopAdjoint: return k_genz_w32<NPART, G, CG, pol::Adjoint<float, GEN>>;
    case kLoopLogWeight: return k_genz_w32<NPART, G, CTAS, pol::Forward<float, GEN, false, dbgz::StepFp32, true>>;
    default:
      if (lower_inf) return k_genz_w32<NPART, G, CTAS, pol::Forward<float, GEN, false, dbgz::StepFp32LowerInf>>;
      return k_genz_w32<NPART, G, CTAS, pol::Forward<float, GEN, false>>;
  }
}

template <int NPART, int G, int CTAS>
int w32_launch(dbgz_problem *p, const PassArgs &pa, double *partials, int64_t n_tiles, int64_t band) {
  dbgz_ctx *ctx = p->ctx;
  const bool adj = pa.kind == kLoopAdjoint;
  const W32Layout<NPART, G> L(pa.d, band);
  DevBuf &ob = adj ? p->w32b_ops : p->w32_ops;
  DBGZ_TRY((w32_operands<NPART, G>(p, adj, band, ob)));
  w32::Params P{};
  w32::Prob &Q = P.pr;
  Q.d = pa.d;
  Q.m = pa.m;
  Q.tiles_per_shift = (pa.m + w32::TS - 1) / w32::TS;
  Q.gen.qmc_type = pa.qmc_type;
  Q.gen.n_bits = pa.n_bits;
  Q.gen.gen_base = pa.gen_base;
  Q.gen.gen_base_dev = pa.gen_base_dev;
  Q.gen.sobol_staged = pa.qmc_type == DBGZ_QMC_SOBOL;
  Q.gen.sobol_first = pa.sobol_first;
  Q.gen.q = (const double *)p->q.p;
  Q.gen.shift64 = (const double *)p->shifts.p;
  Q.gen.shift32 = (const float *)p->shifts32.p;
  Q.gen.V = (const uint32_t *)p->V.p;
  Q.gen.ushift = (const uint64_t *)p->ushifts.p;
  Q.tgt = (const TargetParams32 *)p->tgt32.p;
  const char *base = (const char *)ob.p;
  for (int i = 0; i < 3; ++i) Q.u[i] = (const uint16_t *)(base + (i < NPART ? i : 0) * L.rows_bytes);
  Q.tri = (const float *)(base + L.rows_bytes * NPART);
  Q.ld = L.ld;
  Q.band = band;
  Q.ring_chunks = L.ring_chunks;
  Q.c[0] = pa.c1;
  Q.c[1] = pa.dc1;
  Q.c[2] = 1.0 - pa.c1 - pa.dc1;
  Q.partials = partials;
  P.n_tiles = n_tiles;
  P.tile0 = pa.tile0;
  P.io.N = pa.grad.N;
  P.io.rows = pa.io_rows > 0 ? pa.io_rows : pa.d;
  P.io.y = (float *)pa.grad.y;
  P.io.s = (float *)pa.grad.s;
  P.io.dc = (float *)pa.grad.dc;
  P.io.sbar = (float *)pa.grad.sbar;
  P.io.p = pa.grad.p;
  P.io.ga = pa.grad.ga;
  P.io.gb = pa.grad.gb;
  P.io.gu = pa.grad.gu;
  P.io.dc1 = pa.grad.dc1;
  P.io.tile0 = pa.tile0;
  const int smem = (int)sizeof(w32::Smem<NPART, G>);
  auto kern = pa.qmc_type == DBGZ_QMC_SOBOL ? w32_pick<NPART, G, CTAS, DBGZ_QMC_SOBOL>(pa.kind, p->lower_inf)
                                            : w32_pick<NPART, G, CTAS, DBGZ_QMC_RICHTMYER>(pa.kind, p->lower_inf);
  DBGZ_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int per_sm = 0;
  DBGZ_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, w32::NT, smem));
  if (per_sm < 1) return dbgz_fail(ctx, DBGZ_ERR_CUDA, "FP32 loop: kernel does not fit on an SM");
  const int64_t grid = std::min<int64_t>(n_tiles - pa.tile0, (int64_t)per_sm * ctx->num_sms);
  if (grid < 1) return DBGZ_OK;
  DBGZ_TRY(dbgz_ensure(ctx, p->yws, (size_t)L.slot * grid));
  P.yws = (unsigned char *)p->yws.p;
  P.yws_slot = L.slot;
  if (pa.setup_only) return DBGZ_OK;
  kern<<<(unsigned)grid, w32::NT, smem, ctx->stream>>>(P);
  dbgz_count_launch(ctx);
  DBGZ_CUDA_TRY(ctx, cudaGetLastError());
  return DBGZ_OK;
}

}  // namespace
