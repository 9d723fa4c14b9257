// loop_w32_kernels.cuh -- FP32-class integration loop with one warp per 32
// samples and the contraction on warp-level tensor instructions (launched by
// loop_w32.cu and batch.cu).
//
// What bounds the FP32 loops is the sequential step: about 130 instructions
// in one dependent chain of some 330 cycles, so a scheduler needs four or more
// warps of samples.  The tcgen05 loop (loop_umma.cu) holds two: its partial
// sums take 256 TMEM columns and 32 registers a sample.  Here a warp keeps the
// sums of 32 targets in 4 KB of shared memory and 8 of them in registers, so
// 16 warps fit on an SM, and mma.m16n8k16 (8 cycles of a scheduler, in the
// shadow of the other warps' steps) feeds them without a round trip to
// another warp.  The larger the dimension, the more the contraction weighs:
// mma.sync runs at about a quarter of tcgen05's rate (dbgz_umma_waits has
// the crossover).
//
// One CTA = one tile of 128 samples = four warps of 32.  y-indices run in
// groups of G, each in chunks of 8:
//   * group start: S[32 x G] = Y[:, k0 .. g0) U[k0 .. g0, targets], Y from the
//     CTA's workspace and U^T panels through a two-stage cp.async ring that
//     lies in the S buffer (idle then).  Banded factors: k0 is the first
//     y-index within the band of the group, else 0;
//   * chunk: its sums + the group's own earlier chunks and the chunk's triangle
//     as FP32 FMAs on FP32 y's and coefficients, as the tcgen05 loop does within
//     its blocks of 32 (a chunk's y's take the place of the sums they consumed);
//     the y's that a later group reads go to the workspace as BF16 parts.
//     (With the earlier chunks as BF16 parts too, rms error of the shifts' means
//     against FP64, split BF16: 2.1e-7 at d = 20, 1.9e-7 at 33, geometric mean
//     over d = 8..380 4.3e-7; as FP32 0.8e-7, 0.7e-7, 3.4e-7.  Time with the parts and now: batch of
//     256 problems 20.50 / 20.27 ms, banded d = 4000 pass 10.46 / 10.52, gradient
//     7.81 / 7.70.)
// The tensor unit truncates as it accumulates, so the products of high parts
// have accumulators of their own: their sum is truncated once per 16 y-indices,
// not once per product (relative error of P, batch of d 16..256: 4.7e-6 with
// one accumulator).  Operands are NPART BF16 parts: 2 (hi hi + hi lo + lo hi:
// the split-BF16 mode) or 3 (six products, about 2^-24: FP32 operands' accuracy, for the
// banded loop), from one group to the later ones.  Warps meet once per chunk of
// the ring and per 32 dimensions (their staged constants, copied one block ahead).
#pragma once
#include <type_traits>

#include "internal.cuh"
#include "genz_step.cuh"
#include "loop_simt_kernels.cuh"
#include "policies.cuh"

namespace w32 {

constexpr int TS = 128, NT = 128;
constexpr int SB = 32;  // dimensions per staged block
constexpr int CH = 8;   // y-indices per chunk
constexpr int kTri = 10 * CH * CH;  // FP32 coefficients of a group: its 10 blocks of 8 x 8
__host__ __device__ constexpr int tri_at(int q, int c) { return (q * (q + 1) / 2 + c) * CH * CH; }
constexpr int KC = 16;  // y-indices per ring stage
constexpr int NST = 2;     // stages of the ring
constexpr int kAhead = 1;  // points formed ahead of the steps

// One problem's operands and constants.
struct Prob {
  int64_t d, m, tiles_per_shift;
  dbgz::GenParams gen;
  const TargetParams32 *tgt;
  // per group of 32 y-indices kTri floats: block (q, c), c <= q < 4, at
  // tri_at(q, c): [k * 8 + j] = U[y-index 8 c + k, target of step 8 q + j] (0
  // below the diagonal)
  const float *tri;
  // U^T panels: part p of U[l, t] at u[p][t * ld + l - lofs(group of t)]
  const uint16_t *u[3];
  int64_t ld;
  int64_t band;         // > 0: U[l, t] = 0 for t - l > band
  int64_t ring_chunks;  // chunks of 8 y-indices the workspace holds
  const double *first;  // c1, dc1, up1 in device memory, or null: c
  double c[3];
  double *partials;
};
struct Params {
  Prob pr;
  int64_t n_tiles, tile0;
  unsigned char *yws;  // per CTA: [chunk][warp][part][32 samples][8] BF16
  int64_t yws_slot;    // bytes per CTA
  pol::GradIO<float> io;
};

// first y-index that reaches the targets of group g0 (a multiple of KC)
template <int G>
__host__ __device__ inline int64_t first_k(int64_t g0, int64_t band) {
  const int64_t k = band > 0 ? g0 + 1 - band : 0;
  return k > 0 ? k / KC * KC : 0;
}

// element e of Prob::tri for the factor U (d x d, column-major)
__device__ __forceinline__ float tri_value(const double *U, int64_t d, int64_t e) {
  const int64_t g = e / kTri;
  const int r = (int)(e - g * kTri), blk = r >> 6, k = (r >> 3) & 7, j = r & 7;
  const int q = blk >= 6 ? 3 : blk >= 3 ? 2 : blk >= 1 ? 1 : 0, c = blk - q * (q + 1) / 2;
  const int64_t l = SB * g + 8 * c + k, t = SB * g + 8 * q + j + 1;
  return l < t && t < d ? (float)U[t * d + l] : 0.f;
}

struct Stage {
  pol::Staged<float> sg;
  float tri[kTri];
  uint32_t sob[SB][dbgz::kSobolRow];
};
template <int NPART, int G>
struct Smem {
  static_assert(G == SB, "a staged block holds the coefficients of one group");
  static constexpr int SLOT = 1024;  // a chunk's sums, then its y's: 8 floats a sample
  struct Ring {
    unsigned char y[NST][4][KC / CH][NPART][512];
    unsigned char u[NST][NPART][2][G][16];  // [part][k half][target][8 BF16]
  };
  union {
    unsigned char s[4][G / CH][SLOT];
    Ring ring;
  } u;
  Stage stg[2];
  double red[4];
};

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The products of the parts: every (i, j) with i + j < NPART.
template <int NPART, typename F>
__device__ __forceinline__ void products(F &&f) {
#pragma unroll
  for (int i = 0; i < NPART; ++i)
#pragma unroll
    for (int j = 0; j < NPART; ++j)
      if (i + j < NPART) f(i, j);
}
// A chunk's sums: 8 floats a sample, its two 16-byte halves swapped for every
// other four samples (conflict-free for a sample's own 16-byte loads and for
// an mma fragment's 8-byte ones).  Byte offset of targets t, t + 1 (t even) of
// sample r.
__device__ __forceinline__ uint32_t soff(int t, int r) {
  return (uint32_t)(r * 32 + ((((t >> 2) ^ (r >> 2)) & 1) << 4) + (t & 2) * 4);
}
__device__ __forceinline__ void sts2(uint32_t a, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void lds4(float *x, uint32_t a) {
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t a, const float *x) {
  asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]) : "memory");
}

// two FP32 values in a 64-bit register; c += a b for both, each rounded as fmaf
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &x, float &y) {
  asm("mov.b64 {%0,%1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t &c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// x as BF16 parts of 8 values: word e of part p holds values 2e, 2e + 1
template <int NPART>
__device__ __forceinline__ void split8(const float (&y)[8], uint32_t (&w)[NPART][4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a = y[2 * e], b = y[2 * e + 1];
#pragma unroll
    for (int p = 0; p < NPART; ++p) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
      w[p][e] = *reinterpret_cast<const uint32_t *>(&h);
      if (p + 1 < NPART) {
        const float2 hf = __bfloat1622float2(h);
        a -= hf.x;
        b -= hf.y;
      }
    }
  }
}

template <typename P, typename = void>
struct chunk_redo : std::false_type {};
template <typename P>
struct chunk_redo<P, std::void_t<decltype(P::kChunkRedo)>> : std::bool_constant<P::kChunkRedo> {};

template <int NPART, int G, typename Policy>
__device__ __forceinline__ void tile(const Prob &P, const pol::GradIO<float> &io, Smem<NPART, G> &sm,
                                     unsigned char *Yw, int64_t tile_id) {
  using SM = Smem<NPART, G>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fr = lane >> 2, fk = lane & 3;
  const int64_t d = P.d, nY = d - 1;
  const int64_t k_shift = tile_id / P.tiles_per_shift;
  const int64_t j = (tile_id - k_shift * P.tiles_per_shift) * TS + tid;
  const uint32_t Sa = saddr(&sm.u.s[warp][0][0]);
  // this lane's fragment sums (samples fr + 8 h of the m-tile: +256 h bytes; the
  // other m-tile: +512) and its own sums' halves
  const uint32_t sf = soff(2 * fk, fr), s_lo = soff(0, lane), s_hi = soff(4, lane);
  // ldmatrix row of this lane: matrices (samples 0-7, 8-15) x (first, second chunk)
  const int lm_row = (lane & 7) + ((lane >> 3) & 1) * 8, lm_ch = lane >> 4;
  Policy pl;
  if (P.first)
    pl.tile_begin(P.gen, d, tile_id, P.tiles_per_shift, tid, P.first[0], P.first[1], P.first[2], 0, io);
  else
    pl.tile_begin(P.gen, d, tile_id, P.tiles_per_shift, tid, P.c[0], P.c[1], P.c[2], 0, io);
  const uint64_t base0 = (uint64_t)(P.gen.sobol_first + pl.gen.gen_base + (j - tid));
  const dbgz::SobolLane sob_lane(tid, base0);
  const bool sob_staged = Policy::kSobolTable && pl.gen.sobol_staged;

  // copies of the constants of the block at lb into buffer b (visible after a
  // wait and a barrier)
  auto stage = [&](int b, int64_t lb) {
    Stage &st = sm.stg[b];
    const int nb = (int)(nY - lb < SB ? nY - lb : SB);
    pl.stage_async(st.sg, P.tgt, tid, lb, nb);
    for (int e = tid; e < kTri / 4; e += NT) cp16(saddr(st.tri + 4 * e), P.tri + lb / SB * kTri + 4 * e);
    pol::cp_async_commit();
    if constexpr (Policy::kSobolTable)
      if (sob_staged)
        dbgz::sobol_stage_block(st.sob, P.gen.V, P.gen.ushift + k_shift * (d - 1), dbgz::sobol_mask(P.gen.n_bits),
                                base0, pl.sobol_l0(lb), Policy::kSobolDir, d - 2, nb, tid);
  };
  // this lane's place in the workspace chunk of the next 8 y's (a ring for
  // banded factors)
  unsigned char *yout = Yw + warp * (NPART * 512) + lane * 16;
  const unsigned char *yend = yout + P.ring_chunks * (4 * NPART * 512);
  stage(0, 0);
  pol::cp_async_wait_all();
  __syncthreads();
  int buf = 0;

  for (int64_t g0 = 0; g0 < nY; g0 += G) {
    const int ng = (int)(nY - g0 < (int64_t)G ? nY - g0 : (int64_t)G);
    const int nt = (ng + CH - 1) / CH;
    const bool keep = g0 + G < nY;
    const int64_t k0 = first_k<G>(g0, P.band), lofs = P.band > 0 ? k0 : 0;
    if (g0 > 0) {
      float acc[2][2][G / CH][4];  // [0]: high parts' products, [1]: the others
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int ni = 0; ni < G / CH; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[h][mi][ni][e] = 0.f;
      const int nch = (int)((g0 - k0) / KC);
      // this thread's share of a stage: NPART pieces of each of its warp's two
      // Y chunks (a pair never straddles the workspace's wrap: both sizes are
      // even), and UP pieces of the U panels; sources advance by a stage
      constexpr int NU = G * 2 * NPART, UP = (NU + NT - 1) / NT;
      uint32_t yslot = (uint32_t)(k0 / CH) % (uint32_t)P.ring_chunks;
      // (no rows past the group's last chunk of targets; in it, those past the
      // last target read the last one's, for sums that nobody takes)
      const uint16_t *usrc[UP];
      uint32_t udst[UP];
      bool uval[UP];
#pragma unroll
      for (int e = 0; e < UP; ++e) {
        const int el = tid + NT * e, p = el / (2 * G), q = el % (2 * G), t = q >> 1, h = q & 1;
        const uint16_t *up = NPART > 2 && p > 1 ? P.u[2] : (p == 1 ? P.u[1] : P.u[0]);
        uval[e] = el < NU && t < CH * nt;
        usrc[e] = up + (g0 + 1 + t < d ? g0 + 1 + t : d - 1) * P.ld + (k0 - lofs) + 8 * h;
        udst[e] = saddr(&sm.u.ring.u[0][0][0][0][0]) + (uint32_t)((p * 2 + h) * G + t) * 16;
      }
      const uint32_t ydst = saddr(&sm.u.ring.y[0][warp][0][0][lane * 16]);
      int is = 0, il = 0;  // stage and number of the next chunk to issue
      auto issue = [&]() {
        if (il < nch) {
          const unsigned char *src = Yw + (int64_t)(yslot * 4 + warp) * (NPART * 512) + lane * 16;
#pragma unroll
          for (int h = 0; h < KC / CH; ++h)
#pragma unroll
            for (int p = 0; p < NPART; ++p)
              cp16(ydst + is * (uint32_t)sizeof(sm.u.ring.y[0]) + h * (NPART * 512) + p * 512,
                   src + h * (4 * NPART * 512) + p * 512);
          yslot = yslot + 2 == (uint32_t)P.ring_chunks ? 0u : yslot + 2;
#pragma unroll
          for (int e = 0; e < UP; ++e)
            if (uval[e]) {
              cp16(udst[e] + is * (uint32_t)sizeof(sm.u.ring.u[0]), usrc[e]);
              usrc[e] += KC;
            }
        }
        pol::cp_async_commit();
        ++il;
        is = is + 1 == NST ? 0 : is + 1;
      };
      // (the ring lies in the S buffer: every warp has passed the block
      // barrier of the last group's last chunk)
#pragma unroll
      for (int c = 0; c < NST - 1; ++c) issue();
      const uint32_t ya = saddr(&sm.u.ring.y[0][warp][lm_ch][0][lm_row * 16]);
      const uint32_t ua = saddr(&sm.u.ring.u[0][0][(lane >> 3) & 1][(lane >> 4) * CH + (lane & 7)][0]);
      int s = 0;
      for (int c = 0; c < nch; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
        __syncthreads();
        issue();
        // one m-tile after the other: half the A fragments at a time (with
        // both, three parts spilled)
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          uint32_t a[NPART][4];
#pragma unroll
          for (int p = 0; p < NPART; ++p) ldsm4(a[p], ya + s * (uint32_t)sizeof(sm.u.ring.y[0]) + p * 512 + mi * 256);
#pragma unroll
          for (int n2 = 0; n2 < G / CH; n2 += 2)
            if (n2 < nt) {
              // (targets n2, k half 0), (n2, 1), (n2 + 1, 0), (n2 + 1, 1)
              uint32_t b[NPART][4];
#pragma unroll
              for (int p = 0; p < NPART; ++p)
                ldsm4(b[p], ua + s * (uint32_t)sizeof(sm.u.ring.u[0]) + p * (2 * G * 16) + n2 * (CH * 16));
              products<NPART>([&](int i, int jj) {
                mma16(acc[i + jj > 0][mi][n2], a[i], b[jj][0], b[jj][1]);
                mma16(acc[i + jj > 0][mi][n2 + 1], a[i], b[jj][2], b[jj][3]);
              });
            }
        }
        s = s + 1 == NST ? 0 : s + 1;
      }
      __syncthreads();  // the ring is read: S may be written
#pragma unroll
      for (int ni = 0; ni < G / CH; ++ni)
        if (ni < nt) {
#pragma unroll
          for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              sts2(Sa + ni * SM::SLOT + sf + mi * 512 + h * 256, acc[0][mi][ni][2 * h] + acc[1][mi][ni][2 * h],
                   acc[0][mi][ni][2 * h + 1] + acc[1][mi][ni][2 * h + 1]);
        }
      __syncwarp();
    }
    for (int b0 = 0; b0 < ng; b0 += SB) {
      const int nb = ng - b0 < SB ? ng - b0 : SB;
      const int64_t lb = g0 + b0;
      if (lb + SB < nY) stage(buf ^ 1, lb + SB);
      const Stage &st = sm.stg[buf];
#pragma unroll 1
      for (int i0 = 0; i0 < nb; i0 += CH) {
        const int q = (b0 + i0) / CH;  // chunk of the group
        const int nv = nb - i0;        // valid steps (8 or more: all)
        const uint32_t Sq = Sa + q * SM::SLOT;
        float s[8];
        // (a sample's sums and y's in S are its own lane's)
        if (g0 > 0) {
          lds4(s, Sq + s_lo);
          lds4(s + 4, Sq + s_hi);
        } else {
#pragma unroll
          for (int t = 0; t < 8; ++t) s[t] = 0.f;
        }
        // the group's earlier chunks (paired FMAs: half the issue slots; a copy of the
        // code per chunk: banded pass 10.66 -> 10.52 ms, batch 20.44 -> 20.27)
        if (q > 0) {
          uint64_t s2[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) s2[t] = pack2(s[2 * t], s[2 * t + 1]);
#pragma unroll
          for (int c = 0; c < G / CH - 1; ++c)
            if (c < q) {
              float ye[8];
              lds4(ye, Sa + c * SM::SLOT + s_lo);
              lds4(ye + 4, Sa + c * SM::SLOT + s_hi);
              const ulonglong2 *ur = reinterpret_cast<const ulonglong2 *>(st.tri + tri_at(q, c));
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const uint64_t y2 = pack2(ye[k], ye[k]);
                const ulonglong2 u0 = ur[2 * k], u1 = ur[2 * k + 1];
                fma2(s2[0], y2, u0.x);
                fma2(s2[1], y2, u0.y);
                fma2(s2[2], y2, u1.x);
                fma2(s2[3], y2, u1.y);
              }
            }
#pragma unroll
          for (int t = 0; t < 4; ++t) unpack2(s2[t], s[2 * t], s[2 * t + 1]);
        }
        float ys[8];
        const int64_t l0 = lb + i0;
        pl.chunk_begin(l0, nv);
        // points ahead of the steps: they do not depend on the recursion, and
        // their FP64 and conversion latencies are long
        auto sob_x = [&](int k) -> uint32_t {
          if constexpr (Policy::kSobolTable)
            if (sob_staged) return sob_lane.at(st.sob, i0 + k);
          return 0u;
        };
        auto point = [&](int k) { return pl.point(st.sg, i0 + k, l0 + k, sob_x(k)); };
        typename Policy::Point pt[8];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) pt[k] = point(k);
        auto steps = [&](auto checked, auto fast) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int li = i0 + k;
            float y = 0.f;
            if (!decltype(checked)::value || k < nv) {
              const int64_t l = l0 + k;
              if (k + kAhead < 8) pt[k + kAhead] = point(k + kAhead);
              if constexpr (Policy::kDeferTail)
                y = pl.emit_k_at(st.sg, li, l, k, pt[k]);
              else if constexpr (decltype(fast)::value)
                y = pl.emit_k_fast_at(st.sg, li, l, k, pt[k]);
              else
                y = pl.emit_k(st.sg, li, l, k, sob_x(k));
              const float4 *ur = reinterpret_cast<const float4 *>(st.tri + tri_at(q, q) + k * CH);
              const float4 u0 = ur[0], u1 = ur[1];
              const float uu[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
              for (int t = k; t < 8; ++t) s[t] = fmaf(y, uu[t], s[t]);
              if constexpr (Policy::kDeferTail)
                pl.consume_deferred(st.sg, s[k], li, l, k);
              else
                pl.consume(st.sg, s[k], li, l);
            }
            ys[k] = y;
          }
        };
        auto run = [&](auto fast) {
          if (nv >= 8) steps(std::false_type{}, fast);
          else steps(std::true_type{}, fast);
        };
        if constexpr (chunk_redo<Policy>::value) {
          // as in the tcgen05 loop: without per-step votes, redone with them
          // when a lane's FP32 terms left FP32 range
          float s_save[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) s_save[t] = s[t];
          const auto yb_save = pl.ybar;
          pl.bad = false;
          run(std::true_type{});
          if (__any_sync(0xffffffffu, pl.bad)) {
#pragma unroll
            for (int t = 0; t < 8; ++t) s[t] = s_save[t];
            pl.ybar = yb_save;
            pl.fp64_done = 0u;
            run(std::false_type{});
          }
        } else {
          run(std::false_type{});
        }
        pl.chunk_end(l0, nv);
        if constexpr (Policy::kDeferTail) pl.tail_repair(st.sg, s, i0, l0);
        if (q + 1 < nt) {
          sts4(Sq + s_lo, ys);
          sts4(Sq + s_hi, ys + 4);
        }
        if (keep) {
          uint32_t w[NPART][4];
          split8<NPART>(ys, w);
#pragma unroll
          for (int p = 0; p < NPART; ++p)
            *reinterpret_cast<uint4 *>(yout + p * 512) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
        }
        yout += 4 * NPART * 512;
        if (P.band > 0 && yout == yend) yout -= P.ring_chunks * (4 * NPART * 512);
      }
      // the next block's constants have landed, and this block's are read
      pol::cp_async_wait_all();
      __syncthreads();
      buf ^= 1;
    }
  }
  pl.tile_end(P.tgt, tid, warp, tile_id, j < P.m);
  double pv = pl.tile_value(j < P.m);
  for (int o = 16; o > 0; o >>= 1) pv += __shfl_down_sync(0xffffffffu, pv, o);
  if (lane == 0) sm.red[warp] = pv;
  __syncthreads();
  if (tid == 0) P.partials[tile_id] = ((sm.red[0] + sm.red[1]) + sm.red[2]) + sm.red[3];
}

template <int NPART, int G, int CTAS, typename Policy>
__global__ void __launch_bounds__(NT, CTAS) k_genz_w32(const __grid_constant__ Params P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem<NPART, G> &sm = *reinterpret_cast<Smem<NPART, G> *>(smem_raw);
  unsigned char *Yw = P.yws + (int64_t)blockIdx.x * P.yws_slot;
  for (int64_t t = P.tile0 + blockIdx.x; t < P.n_tiles; t += gridDim.x) tile<NPART, G, Policy>(P.pr, P.io, sm, Yw, t);
}

// Many problems in one launch: work item it is tile it % nt of problem it / nt
// (problems in decreasing dimension), taken from a global counter.
template <int NPART, int G, int CTAS, typename Policy>
__global__ void __launch_bounds__(NT, CTAS)
    k_genz_w32_batch(const Prob *probs, int64_t n_items, int64_t nt, unsigned long long *counter, unsigned char *yws,
                     int64_t yws_slot) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem<NPART, G> &sm = *reinterpret_cast<Smem<NPART, G> *>(smem_raw);
  __shared__ Prob P;
  __shared__ long long cur;
  unsigned char *Yw = yws + (int64_t)blockIdx.x * yws_slot;
  const pol::GradIO<float> io;
  long long loaded = -1;
  for (;;) {
    if (threadIdx.x == 0) cur = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    const long long it = cur;
    if (it >= n_items) break;
    const long long k = it / nt;
    if (k != loaded) {
      static_assert(sizeof(Prob) % 4 == 0, "copied in words");
      for (int e = threadIdx.x; e < (int)(sizeof(Prob) / 4); e += NT)
        reinterpret_cast<uint32_t *>(&P)[e] = reinterpret_cast<const uint32_t *>(probs + k)[e];
      loaded = k;
      __syncthreads();
    }
    tile<NPART, G, Policy>(P, io, sm, Yw, it - k * nt);
  }
}

}  // namespace w32
