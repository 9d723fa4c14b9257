// loop_w32.cu -- the warp-level FP32 loop for dense factors (split BF16): one
// problem, and batches (batch.cu).
#include <vector>

#include "loop_w32_impl.cuh"

namespace {

constexpr int kG = 32, kCtas = 4;

// Operands of every problem of a batch (loop_w32_impl.cuh's k_w32_panels and
// k_w32_tri, for problems blockIdx.y + i gridDim.y).
struct OpsProb {
  const double *U;
  int64_t d, ld, tri_n;
  uint16_t *u0, *u1;
  float *tri;
};
__global__ void k_w32_ops_batch(const OpsProb *probs, int64_t n) {
  for (int64_t k = blockIdx.y; k < n; k += gridDim.y) {
    const OpsProb P = probs[k];
    const int64_t step = (int64_t)gridDim.x * blockDim.x, e0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t e = e0; e < P.d * P.ld; e += step) {
      const int64_t t = e / P.ld, l = e - t * P.ld;
      const double u = l < t ? P.U[t * P.d + l] : 0.0;
      const __nv_bfloat16 h = __double2bfloat16(u);
      P.u0[e] = __bfloat16_as_ushort(h);
      P.u1[e] = __bfloat16_as_ushort(__double2bfloat16(u - (double)__bfloat162float(h)));
    }
    for (int64_t e = e0; e < P.tri_n; e += step) P.tri[e] = w32::tri_value(P.U, P.d, e);
  }
}

auto batch_kernel(int qmc_type) {
  return qmc_type == DBGZ_QMC_SOBOL
             ? w32::k_genz_w32_batch<2, kG, kCtas, pol::Forward<float, DBGZ_QMC_SOBOL, false>>
             : w32::k_genz_w32_batch<2, kG, kCtas, pol::Forward<float, DBGZ_QMC_RICHTMYER, false>>;
}

}  // namespace

int dbgz_loop_w32(dbgz_problem *p, const PassArgs &pa, double *partials, int64_t n_tiles) {
  return w32_launch<2, kG, kCtas>(p, pa, partials, n_tiles, 0);
}

int dbgz_w32_batch_setup(dbgz_ctx *ctx, const UmmaBatchArgs &A, W32BatchPlan **out) {
  *out = nullptr;
  if (A.probs.empty()) return DBGZ_OK;
  const int64_t nsel = (int64_t)A.probs.size();
  W32BatchPlan *B = new W32BatchPlan;
  B->ctx = ctx;
  B->qmc_type = A.qmc_type;
  B->nsel = nsel;
  B->nt = A.tiles_per_shift * A.n_reps;
  B->n_items = nsel * B->nt;
  auto fail = [&](int rc) {
    dbgz_w32_batch_free(B);
    return rc;
  };
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  // operands of problem i at base + off[i]: two panels, then the groups' FP32 coefficients
  std::vector<size_t> off(nsel);
  size_t bytes = 0;
  int64_t slot = 0;
  for (int64_t i = 0; i < nsel; ++i) {
    const W32Layout<2, kG> L(A.dims[A.probs[i]], 0);
    off[i] = bytes;
    bytes += al(2 * L.rows_bytes + sizeof(float) * L.tri_n);
    slot = std::max(slot, L.slot);
  }
  const auto kern = batch_kernel(A.qmc_type);
  const int smem = (int)sizeof(w32::Smem<2, kG>);
  int per_sm = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, w32::NT, smem) != cudaSuccess || per_sm < 1)
    return fail(dbgz_fail(ctx, DBGZ_ERR_CUDA, "FP32 batch loop: kernel does not fit on an SM"));
  B->smem = smem;
  B->grid = std::min<int64_t>(B->n_items, (int64_t)per_sm * ctx->num_sms);
  B->slot = slot;
  const size_t szOps = al(sizeof(OpsProb) * nsel), szProb = al(sizeof(w32::Prob) * nsel);
  int rc = dbgz_ensure(ctx, B->buf, bytes + szOps + szProb + 256 + al((size_t)slot * B->grid));
  if (rc) return fail(rc);
  char *base = (char *)B->buf.p;
  B->d_ops = base + bytes;
  B->d_probs = B->d_ops + szOps;
  B->d_counter = (unsigned long long *)(B->d_probs + szProb);
  B->yws = (unsigned char *)B->d_counter + 256;
  std::vector<OpsProb> ops(nsel);
  std::vector<w32::Prob> probs(nsel);
  for (int64_t i = 0; i < nsel; ++i) {
    const int64_t k = A.probs[i], d = A.dims[k];
    const W32Layout<2, kG> L(d, 0);
    char *o = base + off[i];
    ops[i] = OpsProb{A.dM + A.off2[k], d, L.ld, L.tri_n, (uint16_t *)o, (uint16_t *)(o + L.rows_bytes),
                     (float *)(o + 2 * L.rows_bytes)};
    w32::Prob &Q = probs[i];
    Q = w32::Prob{};
    Q.d = d;
    Q.m = A.m;
    Q.tiles_per_shift = A.tiles_per_shift;
    Q.gen.qmc_type = A.qmc_type;
    Q.gen.n_bits = A.n_bits;
    Q.gen.sobol_first = A.sobol_first;
    Q.gen.q = A.dq;
    Q.gen.shift32 = A.dsh32 ? A.dsh32 + A.offs[k] : nullptr;
    Q.gen.V = A.dV;
    Q.gen.ushift = A.dush ? A.dush + A.offs[k] : nullptr;
    Q.gen.sobol_staged = A.qmc_type == DBGZ_QMC_SOBOL;
    Q.tgt = A.dt32 + A.off1[k];
    Q.tri = ops[i].tri;
    Q.u[0] = ops[i].u0;
    Q.u[1] = Q.u[2] = ops[i].u1;
    Q.ld = L.ld;
    Q.ring_chunks = L.ring_chunks;
    Q.first = A.dfirst + 3 * k;
    Q.partials = A.dpart + A.part_off[k];
  }
  // static tables (pageable sources: the stream is synchronised before they go)
  if (cudaMemcpyAsync(B->d_ops, ops.data(), sizeof(OpsProb) * nsel, cudaMemcpyHostToDevice, ctx->stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(B->d_probs, probs.data(), sizeof(w32::Prob) * nsel, cudaMemcpyHostToDevice, ctx->stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess)
    return fail(dbgz_fail(ctx, DBGZ_ERR_CUDA, "FP32 batch loop: %s", cudaGetErrorString(cudaGetLastError())));
  *out = B;
  return DBGZ_OK;
}

int dbgz_w32_batch_enqueue(W32BatchPlan *B) {
  dbgz_ctx *ctx = B->ctx;
  cudaStream_t st = ctx->stream;
  DBGZ_CUDA_TRY(ctx, cudaMemsetAsync(B->d_counter, 0, sizeof(unsigned long long), st));
  k_w32_ops_batch<<<dim3(8, (unsigned)std::min<int64_t>(B->nsel, 65535)), 256, 0, st>>>((const OpsProb *)B->d_ops,
                                                                                        B->nsel);
  dbgz_count_launch(ctx);
  batch_kernel(B->qmc_type)<<<(unsigned)B->grid, w32::NT, B->smem, st>>>(
      (const w32::Prob *)B->d_probs, B->n_items, B->nt, B->d_counter, B->yws, B->slot);
  dbgz_count_launch(ctx);
  DBGZ_CUDA_TRY(ctx, cudaGetLastError());
  return DBGZ_OK;
}

void dbgz_w32_batch_free(W32BatchPlan *B) {
  if (!B) return;
  dbgz_release(B->buf);
  delete B;
}
