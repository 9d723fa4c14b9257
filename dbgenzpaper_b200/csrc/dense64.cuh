// dense64.cuh -- FP64 dense kernels of the gradient path, written for this
// library: a tiled GEMM that skips the zero blocks of triangular operands
// and writes only the triangle its caller needs, with split-K partial tiles
// summed in a fixed order, and the inverse of an upper-triangular matrix.
//
//   gemm64:   C = op(A) op(B)  (+ C when accumulate), column-major
//             operands; per 64 x 64 output tile the k range is cut to
//             where the operands' triangles can be nonzero, and tiles
//             outside the requested output triangle are not launched.
//   trinv64:  X = U^-1 for U upper triangular (d x d, column-major).
//
// Used by the Cholesky adjoint (chol_adjoint.cu: U Ubar', U^-1 (.) U^-T,
// U'U) and by the FP64 factor gradient dU[l, t] = sum_n y[l][n] (p sbar)[t][n]
// (grad.cu).  No library GEMM.  The products are mma.m8n8k4.f64: the FP64 rate
// is that of scalar FMAs (16 a cycle and scheduler, measured), with an eighth of
// the instructions and a third of the shared-memory reads.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace dense64 {
namespace {  // internal linkage: every translation unit that includes this gets its own copy

constexpr int BM = 64, BN = 64, BK = 8, NST = 4, NT = 256;

enum OutMode {
  kOutFull = 0,         // every C entry
  kOutLowerPhi = 1,     // i > j: v; i == j: v / 2; i < j: 0 (the Phi of the Cholesky adjoint)
  kOutStrictUpper = 2,  // i < j only (other entries untouched)
};

struct GemmArgs {
  int64_t m = 0, n = 0, k = 0;
  const double *A = nullptr;
  int64_t lda = 0;
  const double *B = nullptr;
  int64_t ldb = 0;
  // > 0 (op = transpose only): the operand is stored in tiles of 128 k, element
  // (k, i) at ((k / 128) * rows + i) * 128 + k % 128 (GradIO's layout): the rows
  // a step reads lie on few pages (with rows 1 MB apart the factor gradient at
  // d = 150 took 457 us)
  int64_t a_rows = 0, b_rows = 0;
  double *C = nullptr;
  int64_t ldc = 0;
  // k range per output tile [i0, i1) x [j0, j1): from max(i0 if kmin_row,
  // j0 if kmin_col) to min(i1 if kmax_row, j1 if kmax_col, k)
  int kmin_row = 0, kmin_col = 0, kmax_row = 0, kmax_col = 0;
  int out = kOutFull;
  int accumulate = 0;  // C += product (else C = product)
  // split-K: splits > 1 writes partial tiles [split][tile_i][tile_j][64 x 64]
  // to `partial`, summed by k_gemm64_reduce
  int splits = 1;
  double *partial = nullptr;
};

__device__ __forceinline__ bool tile_needed(const GemmArgs &g, int64_t i0, int64_t i1, int64_t j0, int64_t j1) {
  if (g.out == kOutLowerPhi) return i1 - 1 >= j0;      // some i >= j
  if (g.out == kOutStrictUpper) return i0 < j1 - 1;    // some i < j
  return true;
}

__device__ __forceinline__ void tile_krange(const GemmArgs &g, int64_t i0, int64_t i1, int64_t j0, int64_t j1,
                                            int64_t &k0, int64_t &k1) {
  k0 = 0;
  if (g.kmin_row && i0 > k0) k0 = i0;
  if (g.kmin_col && j0 > k0) k0 = j0;
  k1 = g.k;
  if (g.kmax_row && i1 < k1) k1 = i1;
  if (g.kmax_col && j1 < k1) k1 = j1;
}

__device__ __forceinline__ double out_value(int out, int64_t i, int64_t j, double v, bool &write) {
  write = true;
  if (out == kOutLowerPhi) return i > j ? v : (i == j ? 0.5 * v : 0.0);
  if (out == kOutStrictUpper) write = i < j;
  return v;
}

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
// 8 bytes global -> shared, or zero
__device__ __forceinline__ void cp8(double *dst, const double *src, bool v) {
  const int n = v ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(n)
               : "memory");
}

// One 64 x 64 output tile per CTA (8 warps of 16 x 32), k in steps of 8
// through a four-stage cp.async ring; row strides of 68 doubles make the
// fragment reads conflict-free.
// TA / TB: op(A) = A' / op(B) = B'.
template <bool TA, bool TB>
__global__ void __launch_bounds__(NT) k_gemm64(const GemmArgs g) {
  __shared__ double As[NST][BK][BM + 4];
  __shared__ double Bs[NST][BK][BN + 4];
  const int64_t tiles_n = (g.n + BN - 1) / BN;
  const int64_t ti = blockIdx.x / tiles_n, tj = blockIdx.x % tiles_n;
  const int64_t i0 = ti * BM, j0 = tj * BN;
  const int64_t i1 = i0 + BM < g.m ? i0 + BM : g.m, j1 = j0 + BN < g.n ? j0 + BN : g.n;
  if (!tile_needed(g, i0, i1, j0, j1)) return;
  int64_t k0, k1;
  tile_krange(g, i0, i1, j0, j1, k0, k1);
  // this split's share of the k range, in whole steps
  if (g.splits > 1) {
    const int64_t steps = (k1 > k0 ? k1 - k0 + BK - 1 : 0) / BK;
    const int64_t per = (steps + g.splits - 1) / g.splits;
    const int64_t s0 = k0 + (int64_t)blockIdx.y * per * BK;
    const int64_t s1 = s0 + per * BK;
    k1 = s1 < k1 ? s1 : k1;
    k0 = s0;
  }
  const int tid = threadIdx.x, warp = tid >> 5, fr = (tid & 31) >> 2, fk = tid & 3;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
  double acc[2][4][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int64_t steps = k1 > k0 ? (k1 - k0 + BK - 1) / BK : 0;
  // a thread's elements: (i, k) of the A tile, op N -> i fastest (coalesced), op
  // T -> k fastest; (k, j) of the B tile, op N -> k fastest, op T -> j fastest;
  // offsets from the step's first k
  constexpr int EL = BM * BK / NT;
  int64_t oa[EL], ob[EL];
  int ka[EL], kb[EL];
  bool va[EL], vb[EL];
#pragma unroll
  for (int q = 0; q < EL; ++q) {
    const int e = tid + NT * q;
    const int ai = TA ? e / BK : e % BM, bj = TB ? e % BN : e / BK;
    ka[q] = TA ? e % BK : e / BM;
    kb[q] = TB ? e / BN : e % BK;
    const int64_t gi = i0 + ai, gj = j0 + bj;
    va[q] = gi < i1;
    vb[q] = gj < j1;
    oa[q] = !TA ? gi + ka[q] * g.lda : (g.a_rows > 0 ? gi * 128 : gi * g.lda) + ka[q];
    ob[q] = TB ? gj + kb[q] * g.ldb : (g.b_rows > 0 ? gj * 128 : gj * g.ldb) + kb[q];
  }
  auto load = [&](int64_t step) {
    if (step < steps) {
      const int st = (int)(step % NST);
      const int64_t kk = k0 + step * BK;
      // (a step never straddles a 128-k tile: k0 and 128 are multiples of BK)
      const double *A = g.A + (!TA ? kk * g.lda : (g.a_rows > 0 ? (kk >> 7) * g.a_rows * 128 + (kk & 127) : kk));
      const double *B = g.B + (TB ? kk * g.ldb : (g.b_rows > 0 ? (kk >> 7) * g.b_rows * 128 + (kk & 127) : kk));
#pragma unroll
      for (int q = 0; q < EL; ++q) {
        const int e = tid + NT * q;
        const bool a = va[q] && kk + ka[q] < k1, b = vb[q] && kk + kb[q] < k1;
        cp8(&As[st][ka[q]][TA ? e / BK : e % BM], a ? A + oa[q] : g.A, a);
        cp8(&Bs[st][kb[q]][TB ? e % BN : e / BK], b ? B + ob[q] : g.B, b);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // a warp whose 16 x 32 part is not needed only loads
  const bool mine = i0 + wm < i1 && j0 + wn < j1 &&
                    tile_needed(g, i0 + wm, i0 + wm + 16, j0 + wn, j0 + wn + 32);
#pragma unroll
  for (int p = 0; p < NST - 1; ++p) load(p);
  for (int64_t s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
    __syncthreads();
    load(s + NST - 1);
    const int st = (int)(s % NST);
    if (mine)
#pragma unroll
    for (int k4 = 0; k4 < BK; k4 += 4) {
      double av[2], bv[4];
#pragma unroll
      for (int a = 0; a < 2; ++a) av[a] = As[st][k4 + fk][wm + 8 * a + fr];
#pragma unroll
      for (int b = 0; b < 4; ++b) bv[b] = Bs[st][k4 + fk][wn + 8 * b + fr];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma(acc[a][b][0], acc[a][b][1], av[a], bv[b]);
    }
  }
  if (g.splits > 1) {
    double *pt = g.partial + (((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * BM) * BN;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) pt[(wn + 8 * b + 2 * fk + e) * BM + wm + 8 * a + fr] = acc[a][b][e];
    return;
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t i = i0 + wm + 8 * a + fr, j = j0 + wn + 8 * b + 2 * fk + e;
        if (i >= i1 || j >= j1) continue;
        bool w;
        double v = acc[a][b][e];
        if (g.accumulate) v += g.C[i + j * g.ldc];
        v = out_value(g.out, i, j, v, w);
        if (w) g.C[i + j * g.ldc] = v;
      }
}

// Sum of the split partial tiles in split order, then the output rule
// (blockIdx.y: a part of the tile's entries).
__global__ void k_gemm64_reduce(const GemmArgs g, int64_t n_tiles) {
  const int64_t tiles_n = (g.n + BN - 1) / BN;
  const int64_t tile = blockIdx.x;
  const int64_t ti = tile / tiles_n, tj = tile % tiles_n;
  const int64_t i0 = ti * BM, j0 = tj * BN;
  const int64_t i1 = i0 + BM < g.m ? i0 + BM : g.m, j1 = j0 + BN < g.n ? j0 + BN : g.n;
  if (!tile_needed(g, i0, i1, j0, j1)) return;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < BM * BN; e += blockDim.x * gridDim.y) {
    const int li = e % BM, lj = e / BM;
    const int64_t i = i0 + li, j = j0 + lj;
    if (i >= i1 || j >= j1) continue;
    double v = 0.0;
#pragma unroll 8
    for (int s = 0; s < g.splits; ++s) v += g.partial[((int64_t)s * n_tiles + tile) * BM * BN + e];
    bool w;
    if (g.accumulate) v += g.C[i + j * g.ldc];
    v = out_value(g.out, i, j, v, w);
    if (w) g.C[i + j * g.ldc] = v;
  }
}

// Bytes of partial tiles a split-K launch needs.
inline size_t gemm64_partial_bytes(const GemmArgs &g) {
  if (g.splits <= 1) return 0;
  const int64_t tiles = ((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
  return sizeof(double) * (size_t)g.splits * (size_t)tiles * BM * BN;
}

// Enqueues C = op(A) op(B) on `st` (one launch, or two with split-K).
// Returns the CUDA error of the launches.
template <bool TA, bool TB>
inline cudaError_t gemm64(const GemmArgs &g, cudaStream_t st, int *launches = nullptr) {
  if (g.m <= 0 || g.n <= 0) return cudaSuccess;
  const int64_t tiles = ((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
  k_gemm64<TA, TB><<<dim3((unsigned)tiles, (unsigned)(g.splits > 1 ? g.splits : 1)), NT, 0, st>>>(g);
  if (launches) ++*launches;
  if (g.splits > 1) {
    k_gemm64_reduce<<<dim3((unsigned)tiles, BM * BN / 256), 256, 0, st>>>(g, tiles);
    if (launches) ++*launches;
  }
  return cudaGetLastError();
}

// X = U^-1, U upper triangular (column-major, ld d; the strict lower
// triangle of U is not read), X upper triangular with zeros below the
// diagonal.  One CTA per column c: back substitution of U x = e_c from
// row c upwards, right-looking (after x_r is known, column r of U -- a
// contiguous read -- updates the rows above it); the right-hand side lives
// in shared memory (8 d bytes).
__global__ void k_trinv64(const double *U, int64_t d, double *X) {
  extern __shared__ double rhs[];
  const int64_t c = blockIdx.x;
  for (int64_t i = threadIdx.x; i < d; i += blockDim.x) rhs[i] = i == c ? 1.0 : 0.0;
  __syncthreads();
  for (int64_t r = c; r >= 0; --r) {
    const double xr = rhs[r] / U[r * d + r];
    const double *ur = U + r * d;
    for (int64_t i = threadIdx.x; i < r; i += blockDim.x) rhs[i] = fma(-ur[i], xr, rhs[i]);
    if (threadIdx.x == 0) X[c * d + r] = xr;
    __syncthreads();
  }
  for (int64_t i = c + 1 + threadIdx.x; i < d; i += blockDim.x) X[c * d + i] = 0.0;
}

// The same back substitution with the next column of U loaded into
// registers while the current one is applied, and one barrier per step:
// every thread forms x_r itself (the same operation on the same operands),
// so the step's only exchange is the right-hand side in shared memory.
// Thread t owns rows t + 128 q, q < Q (d <= 128 Q).
template <int Q>
__global__ void __launch_bounds__(128) k_trinv64_pf(const double *U, int64_t d, double *X) {
  extern __shared__ double rhs[];
  const int64_t c = blockIdx.x;
  const int tid = threadIdx.x;
  for (int64_t i = tid; i < d; i += 128) rhs[i] = i == c ? 1.0 : 0.0;
  double ucur[Q], unext[Q];
  // x_r = rhs_r * (1 / U_rr): the reciprocal of the next step's diagonal is
  // formed while the current step runs, so the chain of steps carries a
  // multiplication, not a division (within an ulp of rhs_r / U_rr)
  double dcur = 1.0 / U[c * d + c], dnext = 1.0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int64_t i = tid + 128 * q;
    ucur[q] = i < c ? U[c * d + i] : 0.0;
  }
  __syncthreads();
  for (int64_t r = c; r >= 0; --r) {
    if (r > 0) {
      const double *un = U + (r - 1) * d;
      dnext = 1.0 / un[r - 1];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int64_t i = tid + 128 * q;
        unext[q] = i < r - 1 ? un[i] : 0.0;
      }
    }
    const double xr = rhs[r] * dcur;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t i = tid + 128 * q;
      if (i < r) rhs[i] = fma(-ucur[q], xr, rhs[i]);
    }
    if (tid == 0) X[c * d + r] = xr;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) ucur[q] = unext[q];
    dcur = dnext;
  }
  for (int64_t i = c + 1 + tid; i < d; i += 128) X[c * d + i] = 0.0;
}

inline size_t trinv64_smem(int64_t d) { return sizeof(double) * (size_t)d; }

template <typename K>
inline cudaError_t trinv64_launch(K kern, const double *U, int64_t d, double *X, cudaStream_t st) {
  const size_t smem = trinv64_smem(d);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kern<<<(unsigned)d, 128, smem, st>>>(U, d, X);
  return cudaGetLastError();
}

inline cudaError_t trinv64(const double *U, int64_t d, double *X, cudaStream_t st, int *launches = nullptr) {
  if (launches) ++*launches;
  if (d <= 128 * 2) return trinv64_launch(k_trinv64_pf<2>, U, d, X, st);
  if (d <= 128 * 4) return trinv64_launch(k_trinv64_pf<4>, U, d, X, st);
  if (d <= 128 * 8) return trinv64_launch(k_trinv64_pf<8>, U, d, X, st);
  if (d <= 128 * 16) return trinv64_launch(k_trinv64_pf<16>, U, d, X, st);
  return trinv64_launch(k_trinv64, U, d, X, st);
}

}  // namespace
}  // namespace dense64
