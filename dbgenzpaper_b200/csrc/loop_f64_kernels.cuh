// loop_f64_kernels.cuh -- device code of the FP64 integration loop (launched
// by loop_simt.cu, batch.cu and noalloc.cu).
//
// The FP64 units bound this loop: one warp-wide FMA takes 2 cycles of a
// scheduler, as scalar DFMAs or inside mma.m8n8k4.f64 (16 cycles for 8 of
// them; measured, both share one pipe).  The mma form is used for every
// contraction because it needs an eighth of the issue slots and a twelfth of
// the shared-memory reads, which leaves both to the special functions.
//
// One CTA = one tile of 128 samples = four warps of 32 samples, every thread
// one sample.  y-indices run in groups of G (their targets are the indices + 1):
//   * S[32 x G] of a warp = Y[:, k0 .. g0) U[k0 .. g0, targets]: 4 x G/8 mma
//     tiles in registers, Y and U staged in chunks of 8 y-indices through a
//     cp.async ring that lies in the S buffer, idle during this phase.  Banded
//     factors: k0 is the first y-index within the band of the group, else 0.
//     G = 32 with 16 warps an SM measured faster than G = 64 with 12 (d = 500:
//     3.60 against 3.84 ms; equal at d = 1000, where its sweeps read Y twice
//     as often; gradient at d = 150 1.82 against 2.00 ms);
//   * in the group, sub-blocks of 8 targets: the sums get the contributions
//     of the group's earlier y's by mma (the y's take the places of the sums
//     they consumed, so the same buffer is the A operand), then 8 sequential
//     steps, one thread per sample, with the sub-block's triangle as FMAs on
//     8 registers that shift by one a step (static indices in a rolled loop:
//     an unrolled one would not fit the instruction cache).
// Warps only meet where they share staged data: per chunk of the sweep and
// per 32 dimensions (whose constants are copied one block ahead).
#pragma once
#include "internal.cuh"
#include "genz_step.cuh"
#include "policies.cuh"
#include "loop_simt_kernels.cuh"

namespace f64 {

constexpr int TS = 128;  // samples per tile
constexpr int NT = 128;  // threads per CTA
constexpr int G = 32;    // y-indices per group
constexpr int SB = 32;   // y-indices per staged block
constexpr int KC = 8;    // y-indices per chunk of the sweep
constexpr int NST = 3;   // stages of the sweep's ring

using Params = simt::SimtParams<double>;

struct Stage {
  pol::Staged<double> sg;
  double tri[SB / 8][8][8];  // [sub-block][k][j] = U[l0 + k, target of step k + j]
  uint32_t sob[SB][dbgz::kSobolRow];
};
struct Smem {
  union {
    double S[4][G][32];  // [warp][target, later y-index][sample ^ swizzle]
    struct {
      double Y[NST][4][KC][32];
      double U[NST][G][KC + 4];  // row stride 12: conflict-free B fragments
    } ring;
  } u;
  Stage stg[2];
  double red[NT / 32];
  dbgz::NormTab tab;
};

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
// sample `row` of row t of a [t][32] buffer: rows 4 apart in the low bits of
// t, so that an A fragment (8 samples x 4 rows) touches every bank once
__device__ __forceinline__ int swz(int t, int row) { return t * 32 + (row ^ ((t & 3) << 2)); }

// One tile of 128 samples of the problem P (all NT threads; Yw is the CTA's
// slot of the Y workspace, [y-index][sample], of which only indices that a
// later group reads are written).
template <typename Policy>
__device__ __forceinline__ void tile(const Params &P, Smem &sm, double *Yw, int64_t tile_id) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fr = lane >> 2, fk = lane & 3;  // fragment row (or column) and k
  const int64_t d = P.d, nY = d - 1;
  const int64_t k_shift = tile_id / P.tiles_per_shift;
  const int64_t j = (tile_id - k_shift * P.tiles_per_shift) * TS + tid;
  double *S = &sm.u.S[warp][0][0];
  Policy pl;
  pl.set_tab(&sm.tab);
  pl.tile_begin(P.gen, d, tile_id, P.tiles_per_shift, tid, P.c1, P.dc1, P.up1, P.cdf_form, P.io);
  const uint64_t base0 = (uint64_t)(P.gen.sobol_first + pl.gen.gen_base + (j - tid));
  const dbgz::SobolLane sob_lane(tid, base0);
  pl.state_begin();
  // copies of the constants of the block at lb into buffer b (visible after a
  // wait and a barrier)
  auto stage = [&](int b, int64_t lb) {
    Stage &st = sm.stg[b];
    const int nb = (int)(nY - lb < SB ? nY - lb : SB);
    pl.stage_async(st.sg, P.tgt, tid, lb, nb);
#pragma unroll
    for (int e = tid; e < SB * 8; e += NT) {
      const int li = e >> 3, jj = e & 7, kk = li & 7;
      const bool v = kk + jj < 8 && li + jj < nb;
      pol::cp_async_or_zero<8>(&st.tri[0][0][0] + e, v ? P.U + (lb + li + jj + 1) * d + lb + li : P.U, v);
    }
    pol::cp_async_commit();
    if constexpr (Policy::kSobolTable)
      if (pl.gen.sobol_staged)
        dbgz::sobol_stage_block(st.sob, P.gen.V, P.gen.ushift + k_shift * (d - 1), dbgz::sobol_mask(P.gen.n_bits),
                                base0, pl.sobol_l0(lb), Policy::kSobolDir, d - 2, nb, tid);
  };
  // this sample's place in the workspace row of the next y (a ring of P.ring
  // rows for banded factors, a multiple of 8)
  double *yout = Yw + tid;
  const double *yend = yout + P.ring * TS;
  stage(0, 0);
  pol::cp_async_wait_all();
  __syncthreads();
  int buf = 0;

  for (int64_t g0 = 0; g0 < nY; g0 += G) {
    const int ng = (int)(nY - g0 < (int64_t)G ? nY - g0 : (int64_t)G);
    const int nt = (ng + 7) >> 3;
    const bool keep = g0 + G < nY;  // a later group reads this group's y's
    if (g0 > 0) {
      // ---- S = Y[:, 0 .. g0) U[0 .. g0, the group's targets] ----
      double acc[4][G / 8][2];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < G / 8; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
      const int64_t k0 = P.band > 0 && g0 + 1 > P.band ? (g0 + 1 - P.band) / KC * KC : 0;
      const int nch = (int)((g0 - k0) / KC);
      // this thread's share of a chunk: four 16-byte pieces of its warp's Y rows
      // and UP coefficients; sources advance by a chunk.  (No rows past the
      // group's last 8 targets; in those, rows past the last target read the
      // last one's, for sums that nobody takes.)
      constexpr int UP = G * KC / NT;
      const double *ysrc = Yw + (P.band > 0 ? k0 % P.ring : 0) * TS + 32 * warp;
      const double *usrc[UP];
      uint32_t ydst[KC / 2], udst[UP];
#pragma unroll
      for (int e = 0; e < KC / 2; ++e) {
        const int kk = (lane + 32 * e) >> 4, row = 2 * (lane & 15);
        ydst[e] = (uint32_t)__cvta_generic_to_shared(&sm.u.ring.Y[0][warp][0][0] + swz(kk, row));
      }
#pragma unroll
      for (int e = 0; e < UP; ++e) {
        const int t = (tid + NT * e) >> 3, kk = tid & 7;
        usrc[e] = P.U + (g0 + 1 + t < d ? g0 + 1 + t : d - 1) * d + k0 + kk;
        udst[e] = (uint32_t)__cvta_generic_to_shared(&sm.u.ring.U[0][t][kk]);
      }
      int is = 0, ich = 0;  // stage and number of the next chunk to issue
      auto issue = [&]() {
        if (ich < nch) {
          const double *ys = ysrc + (lane >> 4) * TS + 2 * (lane & 15);
#pragma unroll
          for (int e = 0; e < KC / 2; ++e)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             ydst[e] + is * (uint32_t)sizeof(sm.u.ring.Y[0])),
                         "l"(ys + 2 * e * TS)
                         : "memory");
          ysrc += KC * TS;
          if (ysrc == yend - tid + 32 * warp) ysrc -= P.ring * TS;
#pragma unroll
          for (int e = 0; e < UP; ++e) {
            if (((tid + NT * e) >> 3) < 8 * nt)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                               udst[e] + is * (uint32_t)sizeof(sm.u.ring.U[0])),
                           "l"(usrc[e])
                           : "memory");
            usrc[e] += KC;
          }
        }
        pol::cp_async_commit();
        ++ich;
        is = is + 1 == NST ? 0 : is + 1;
      };
      // (the ring lies in the S buffer: every warp has passed the block
      // barrier of the last group)
#pragma unroll
      for (int ch = 0; ch < NST - 1; ++ch) issue();
      int rs = 0;
      for (int ch = 0; ch < nch; ++ch) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
        __syncthreads();  // chunk ch has landed for all; the stage of chunk ch - 1 is free
        issue();
        const double *Ys = &sm.u.ring.Y[rs][warp][0][0];
        const double(*Us)[KC + 4] = sm.u.ring.U[rs];
#pragma unroll
        for (int k4 = 0; k4 < KC / 4; ++k4) {
          double av[4];
#pragma unroll
          for (int mi = 0; mi < 4; ++mi) av[mi] = Ys[swz(4 * k4 + fk, 8 * mi + fr)];
#pragma unroll
          for (int ni = 0; ni < G / 8; ++ni)
            if (ni < nt) {
              const double bv = Us[8 * ni + fr][4 * k4 + fk];
#pragma unroll
              for (int mi = 0; mi < 4; ++mi) dmma(acc[mi][ni][0], acc[mi][ni][1], av[mi], bv);
            }
        }
        rs = rs + 1 == NST ? 0 : rs + 1;
      }
      __syncthreads();  // the ring is read: S may be written
#pragma unroll
      for (int ni = 0; ni < G / 8; ++ni)
        if (ni < nt) {
#pragma unroll
          for (int mi = 0; mi < 4; ++mi) {
            S[swz(8 * ni + 2 * fk, 8 * mi + fr)] = acc[mi][ni][0];
            S[swz(8 * ni + 2 * fk + 1, 8 * mi + fr)] = acc[mi][ni][1];
          }
        }
      __syncwarp();
    }
    // ---- sequential steps, 32 dimensions staged at a time ----
    for (int b0 = 0; b0 < ng; b0 += SB) {
      const int nb = ng - b0 < SB ? ng - b0 : SB;
      const int64_t lb = g0 + b0;
      if (lb + SB < nY) stage(buf ^ 1, lb + SB);
      const Stage &st = sm.stg[buf];
      // the tent-transformed point of step li, formed one step ahead
      auto point = [&](int li) -> double {
        uint32_t xs = 0u;
        if constexpr (Policy::kSobolTable)
          if (pl.gen.sobol_staged) xs = sob_lane.at(st.sob, li);
        return pl.point(st.sg, li, lb + li, xs);
      };
      double w = point(0);
      for (int i0 = 0; i0 < nb; i0 += 8) {
        const int q8 = b0 + i0;  // the sub-block's first target in the group
        const int nv = nb - i0 < 8 ? nb - i0 : 8;
        if (q8 > 0) {
          double c[4][2];
#pragma unroll
          for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int e = 0; e < 2; ++e) c[mi][e] = g0 > 0 ? S[swz(q8 + 2 * fk + e, 8 * mi + fr)] : 0.0;
          const int64_t tr = g0 + q8 + 1 + fr;  // (past the last target: its sums are not taken)
          const double *Ut = P.U + (tr < d ? tr : d - 1) * d + g0 + fk;
          // 8 y's (two k steps) a round; the next round's coefficients are
          // loaded while this one's products run
          double b0v = __ldg(Ut), b1v = __ldg(Ut + 4);
          for (int kk = 0; kk < q8; kk += 8) {
            const double c0v = b0v, c1v = b1v;
            if (kk + 8 < q8) {
              b0v = __ldg(Ut + kk + 8);
              b1v = __ldg(Ut + kk + 12);
            }
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) dmma(c[mi][0], c[mi][1], S[swz(kk + fk, 8 * mi + fr)], c0v);
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) dmma(c[mi][0], c[mi][1], S[swz(kk + 4 + fk, 8 * mi + fr)], c1v);
          }
#pragma unroll
          for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int e = 0; e < 2; ++e) S[swz(q8 + 2 * fk + e, 8 * mi + fr)] = c[mi][e];
          __syncwarp();
        }
        double s[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) s[t] = (g0 > 0 || q8 > 0) ? S[swz(q8 + t, lane)] : 0.0;
#pragma unroll 1
        for (int k = 0; k < nv; ++k) {
          const int li = i0 + k;
          const int64_t l = lb + li;
          const double2 *tr = reinterpret_cast<const double2 *>(&st.tri[i0 >> 3][k][0]);
          const double2 t0 = tr[0], t1 = tr[1], t2 = tr[2], t3 = tr[3];
          const double wn = point(li + 1 < nb ? li + 1 : li);
          const double y = pl.emit_next(st.sg, li, l, w);
          w = wn;
          S[swz(q8 + k, lane)] = y;
          if (keep) yout[k * TS] = y;
          const double s0 = fma(y, t0.x, s[0]);
          s[0] = fma(y, t0.y, s[1]);
          s[1] = fma(y, t1.x, s[2]);
          s[2] = fma(y, t1.y, s[3]);
          s[3] = fma(y, t2.x, s[4]);
          s[4] = fma(y, t2.y, s[5]);
          s[5] = fma(y, t3.x, s[6]);
          s[6] = fma(y, t3.y, s[7]);
          pl.consume(st.sg, s0, li, l);
        }
        // a partial sub-block (the problem's last) leaves unused rows: no later mma reads them
        yout += 8 * TS;
        if (yout == yend) yout -= P.ring * TS;
        __syncwarp();
      }
      // the next block's constants have landed, and this block's are read
      pol::cp_async_wait_all();
      __syncthreads();
      buf ^= 1;
    }
  }
  // ---- per-tile end and sum of p (fixed order) ----
  pl.tile_end(P.tgt, tid, 0, tile_id, j < P.m);
  double pv = pl.tile_value(j < P.m);
  for (int o = 16; o > 0; o >>= 1) pv += __shfl_down_sync(0xffffffffu, pv, o);
  if (lane == 0) sm.red[warp] = pv;
  __syncthreads();
  if (tid == 0) P.partials[tile_id] = ((sm.red[0] + sm.red[1]) + sm.red[2]) + sm.red[3];
  __syncthreads();
}

template <typename Policy>
__global__ void __launch_bounds__(NT, 4) k_genz_f64(const __grid_constant__ Params P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  dbgz::norm_tab_load(sm.tab, threadIdx.x, NT);
  __syncthreads();
  double *Yw = P.yws + (int64_t)blockIdx.x * P.Dp * TS;
  for (int64_t t = P.tile0 + blockIdx.x; t < P.n_tiles; t += gridDim.x) tile<Policy>(P, sm, Yw, t);
}

// Many problems in one launch, work items from a global counter (as
// simt::k_genz_simt_batch).
template <typename Policy>
__global__ void __launch_bounds__(NT, 4)
    k_genz_f64_batch(const Params *params, const simt::BatchItem *items, int64_t n_items, unsigned long long *counter,
                     double *yws, int64_t Dp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  dbgz::norm_tab_load(sm.tab, threadIdx.x, NT);
  __syncthreads();
  __shared__ Params Ps;
  __shared__ long long cur;
  double *Yw = yws + (int64_t)blockIdx.x * Dp * TS;
  for (;;) {
    if (threadIdx.x == 0) {
      cur = (long long)atomicAdd(counter, 1ull);
      if (cur < n_items) Ps = params[items[cur].prob];
    }
    __syncthreads();
    const long long it = cur;
    if (it >= n_items) break;
    const simt::BatchItem bi = items[it];
    for (int64_t t = bi.tile0; t < (int64_t)bi.tile0 + bi.ntiles; ++t) tile<Policy>(Ps, sm, Yw, t);
    __syncthreads();
  }
}

}  // namespace f64
