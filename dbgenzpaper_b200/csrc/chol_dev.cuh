// chol_dev.cuh -- CTA-level device code of the pivoted blocked Cholesky,
// shared by the one-problem kernels (chol.cu) and the batched factorisation
// (batch.cu): one Genz pivot block and one Schur-update tile.  Arithmetic
// contract as in chol.cu: every sum is one ascending fma chain, every other
// operation one IEEE operation (detmath.h), so all callers give the same
// bits.
#pragma once
#include <cfloat>
#include <cstdint>

#include "detmath.h"

namespace cholk {

// The order findmin/argmin use (Base.isgreater: NaN lowest, -0.0 below +0.0,
// then by value) as an unsigned key: NaN -> 0, otherwise the IEEE bits made
// monotone (negative values complemented, non-negative ones with the sign bit
// set), so -0.0 sorts below +0.0 and equal values give equal keys.  The
// largest key, +inf's, is below ~0, which marks "no candidate".
__device__ __forceinline__ unsigned long long argmin_key(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  if (x != x) return 0ull;
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// The warp's least key and, among the lanes that hold it, the least index
// (ties go to the first candidate, as findmin's do): three warp
// min-reductions on 32-bit words, no compare-and-branch tree.  Lanes without a
// candidate pass key ~0 and index ~0.
__device__ __forceinline__ void warp_argmin(unsigned long long &key, unsigned &idx) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
  idx = __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? idx : 0xffffffffu);
  key = ((unsigned long long)mh << 32) | ml;
}

// One bs1 block [i0, i1] of cholesky_genz! inside the bs2 panel ending at
// ii1 (0-based, inclusive), src/cholesky.jl:494-572.  One CTA of up to
// 1024 threads (any multiple of 32).
__device__ __forceinline__ void genz_block_dev(double *M, int64_t n, double *a, double *b, double *dvec,
                                               double *svec, double *ovec, int64_t *perm, int64_t i0,
                                               int64_t i1, int64_t ii1, const double *eps0_ptr, int64_t *rank) {
  __shared__ unsigned long long red_k[32];
  __shared__ unsigned red_t[32];
  __shared__ int64_t sh_im;
  __shared__ double sh_mii, sh_yi;
  __shared__ int sh_stop;
  const double c2 = dm_div(1.0, dm_sqrt(2.0));
  const double is2pi = dm_div(2.0, dm_sqrt(dm_mul(2.0, M_PI)));
  const double eps0 = eps0_ptr[0];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (rank[0] < n) return;  // an earlier block already stopped
  for (int64_t k = i0 + tid; k <= ii1; k += blockDim.x) dvec[k] = 0.0;
  __syncthreads();
  for (int64_t i = i0; i <= i1; ++i) {
    // pivot scores :500-512, then argmin :514
    unsigned long long key = ~0ull;  // this thread's least key, at its first position
    unsigned pos = ~0u;
    for (int64_t k = i + tid; k <= ii1; k += blockDim.x) {
      double m_kk = dm_sub(M[k * n + k], dvec[k]);
      m_kk = m_kk < 0 ? 0.0 : dm_sqrt(m_kk);
      double a_k = dm_mul(dm_div(dm_sub(a[k], svec[k]), m_kk), c2);
      double b_k = dm_mul(dm_div(dm_sub(b[k], svec[k]), m_kk), c2);
      double o = dm_sub(det_erf(b_k), det_erf(a_k));
      ovec[k] = o;
      const unsigned long long ko = argmin_key(o);
      if (ko < key) {
        key = ko;
        pos = (unsigned)(k - i0);
      }
    }
    warp_argmin(key, pos);
    if (lane == 0) {
      red_k[wid] = key;
      red_t[wid] = pos;
    }
    __syncthreads();
    if (wid == 0) {
      const int nw = (int)(blockDim.x >> 5);
      key = lane < nw ? red_k[lane] : ~0ull;
      pos = lane < nw ? red_t[lane] : ~0u;
      warp_argmin(key, pos);
    }
    if (tid == 0) {
      const int64_t im = i0 + (int64_t)pos;
      double d_ii = ovec[im];
      double m_ii = dm_sub(M[im * n + im], dvec[im]);
      if (im != i) {  // :518-523
        int64_t tp = perm[i]; perm[i] = perm[im]; perm[im] = tp;
        double t;
        t = dvec[im]; dvec[im] = dvec[i]; dvec[i] = t;
        t = svec[im]; svec[im] = svec[i]; svec[i] = t;
        t = a[im]; a[im] = a[i]; a[i] = t;
        t = b[im]; b[im] = b[i]; b[i] = t;
      }
      sh_im = im;
      sh_mii = m_ii;
      sh_yi = d_ii;  // carried to the y_i step
    }
    __syncthreads();
    const int64_t im = sh_im;
    if (im != i) {  // :525-530: rows over columns i0..n, then full columns
      for (int64_t k = i0 + tid; k < n; k += blockDim.x) {
        double t = M[k * n + i];
        M[k * n + i] = M[k * n + im];
        M[k * n + im] = t;
      }
      __syncthreads();
      for (int64_t k = tid; k < n; k += blockDim.x) {
        double t = M[i * n + k];
        M[i * n + k] = M[im * n + k];
        M[im * n + k] = t;
      }
      __syncthreads();
    }
    if (tid == 0) {
      double m_ii = sh_mii;
      double d_ii = sh_yi;
      int stop = 0;
      if (m_ii > eps0) {
        m_ii = dm_sqrt(m_ii);
      } else {
        rank[0] = i;  // 0-based i == reference's i - 1
        stop = 1;
      }
      if (!stop) {
        M[i * n + i] = m_ii;
        double a_norm = dm_div(dm_sub(a[i], svec[i]), m_ii);
        double b_norm = dm_div(dm_sub(b[i], svec[i]), m_ii);
        double ea = det_exp(dm_div(-dm_mul(a_norm, a_norm), 2.0));
        double eb = det_exp(dm_div(-dm_mul(b_norm, b_norm), 2.0));
        sh_yi = dm_div(dm_mul(dm_sub(ea, eb), is2pi), d_ii);
        sh_mii = m_ii;
      }
      sh_stop = stop;
    }
    __syncthreads();
    if (sh_stop) return;
    const double m_ii = sh_mii, y_i = sh_yi;
    if (i == i0) {  // :547-554
      for (int64_t j = i + 1 + tid; j <= ii1; j += blockDim.x) {
        double m_ij = dm_div(M[j * n + i], m_ii);
        M[j * n + i] = m_ij;
        M[i * n + j] = m_ij;
        dvec[j] = dm_add(dvec[j], dm_mul(m_ij, m_ij));
        svec[j] = dm_add(svec[j], dm_mul(y_i, m_ij));
      }
    } else if (i < ii1) {  // :555-570
      for (int64_t j = i + 1 + tid; j <= ii1; j += blockDim.x) {
        double acc = 0.0;
        for (int64_t l = i0; l <= i - 1; ++l) acc = dm_fma(M[l * n + j], M[i * n + l], acc);
        double m_ij = dm_div(dm_sub(M[i * n + j], acc), m_ii);
        M[j * n + i] = m_ij;
        M[i * n + j] = m_ij;
        dvec[j] = dm_add(dvec[j], dm_mul(m_ij, m_ij));
        svec[j] = dm_add(svec[j], dm_mul(y_i, m_ij));
      }
    }
    __syncthreads();
  }
}

// genz_block_dev with the panel's per-candidate vectors held in shared
// memory for the whole block: dvec, svec, a, b, perm and the diagonal of M
// over [i0, ii1] (sh: 7 (ii1 - i0 + 1) words, see genz_block_smem_bytes).
// The pivot step's serial part (argmin, swaps, the pivot's own terms) then
// makes no global round trips; M's rows and columns stay in global memory.
// Same operations in the same order as genz_block_dev: the same bits.
__host__ __device__ inline size_t genz_block_smem_bytes(int64_t panel_len) { return (size_t)56 * panel_len; }

__device__ __forceinline__ void genz_block_smem(double *M, int64_t n, double *a, double *b, double *dvec,
                                                double *svec, int64_t *perm, int64_t i0, int64_t i1, int64_t ii1,
                                                const double *eps0_ptr, int64_t *rank, double *sh) {
  __shared__ unsigned long long red_k[32];
  __shared__ unsigned red_t[32];
  __shared__ int64_t sh_im;
  __shared__ double sh_mii, sh_yi;
  __shared__ int sh_stop;
  const double c2 = dm_div(1.0, dm_sqrt(2.0));
  const double is2pi = dm_div(2.0, dm_sqrt(dm_mul(2.0, M_PI)));
  const double eps0 = eps0_ptr[0];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (rank[0] < n) return;  // an earlier block already stopped
  const int64_t len = ii1 - i0 + 1;
  double *s_d = sh, *s_s = sh + len, *s_a = sh + 2 * len, *s_b = sh + 3 * len, *s_g = sh + 4 * len,
         *s_o = sh + 5 * len;
  int64_t *s_p = reinterpret_cast<int64_t *>(sh + 6 * len);
  for (int64_t k = tid; k < len; k += blockDim.x) {
    const int64_t g = i0 + k;
    s_d[k] = 0.0;
    s_s[k] = svec[g];
    s_a[k] = a[g];
    s_b[k] = b[g];
    s_g[k] = M[g * n + g];
    s_p[k] = perm[g];
  }
  __syncthreads();
  auto write_back = [&]() {
    __syncthreads();
    for (int64_t k = tid; k < len; k += blockDim.x) {
      const int64_t g = i0 + k;
      dvec[g] = s_d[k];
      svec[g] = s_s[k];
      a[g] = s_a[k];
      b[g] = s_b[k];
      perm[g] = s_p[k];
    }
  };
  for (int64_t i = i0; i <= i1; ++i) {
    // pivot scores :500-512, then argmin :514
    unsigned long long key = ~0ull;  // this thread's least key, at its first position
    unsigned pos = ~0u;
    for (int64_t k = i + tid; k <= ii1; k += blockDim.x) {
      const int64_t q = k - i0;
      double m_kk = dm_sub(s_g[q], s_d[q]);
      m_kk = m_kk < 0 ? 0.0 : dm_sqrt(m_kk);
      double a_k = dm_mul(dm_div(dm_sub(s_a[q], s_s[q]), m_kk), c2);
      double b_k = dm_mul(dm_div(dm_sub(s_b[q], s_s[q]), m_kk), c2);
      double o = dm_sub(det_erf(b_k), det_erf(a_k));
      s_o[q] = o;
      const unsigned long long ko = argmin_key(o);
      if (ko < key) {
        key = ko;
        pos = (unsigned)q;
      }
    }
    warp_argmin(key, pos);
    if (lane == 0) {
      red_k[wid] = key;
      red_t[wid] = pos;
    }
    __syncthreads();
    if (wid == 0) {
      // the warps' minima reduced by warp 0 (the key order with the position
      // as tie-break is a strict total order: the same pivot in any grouping)
      const int nw = (int)(blockDim.x >> 5);
      key = lane < nw ? red_k[lane] : ~0ull;
      pos = lane < nw ? red_t[lane] : ~0u;
      warp_argmin(key, pos);
      const int64_t im = i0 + (int64_t)pos;
      if (lane == 0) {
      const int64_t qi = i - i0, qm = im - i0;
      double d_ii = s_o[qm];
      double m_ii = dm_sub(s_g[qm], s_d[qm]);
      if (im != i) {  // :518-523 (and the diagonal, which the row/column swap moves)
        int64_t tp = s_p[qi]; s_p[qi] = s_p[qm]; s_p[qm] = tp;
        double t;
        t = s_d[qm]; s_d[qm] = s_d[qi]; s_d[qi] = t;
        t = s_s[qm]; s_s[qm] = s_s[qi]; s_s[qi] = t;
        t = s_a[qm]; s_a[qm] = s_a[qi]; s_a[qi] = t;
        t = s_b[qm]; s_b[qm] = s_b[qi]; s_b[qi] = t;
        t = s_g[qm]; s_g[qm] = s_g[qi]; s_g[qi] = t;
      }
      sh_im = im;
      sh_mii = m_ii;
      sh_yi = d_ii;  // carried to the y_i step
      }
    }
    __syncthreads();
    const int64_t im = sh_im;
    // the y_i step (:533-546) by the block's last thread, which has no element
    // of the swap below when n < blockDim: its arithmetic overlaps the swap,
    // its write of the diagonal waits for it (same operations as in order)
    const bool yt = tid == (int)blockDim.x - 1;
    double y_mii = 0.0;
    int y_stop = 0;
    if (yt) {
      double m_ii = sh_mii;
      double d_ii = sh_yi;
      if (m_ii > eps0) {
        m_ii = dm_sqrt(m_ii);
      } else {
        rank[0] = i;  // 0-based i == reference's i - 1
        y_stop = 1;
      }
      if (!y_stop) {
        const int64_t qi = i - i0;
        double a_norm = dm_div(dm_sub(s_a[qi], s_s[qi]), m_ii);
        double b_norm = dm_div(dm_sub(s_b[qi], s_s[qi]), m_ii);
        double ea = det_exp(dm_div(-dm_mul(a_norm, a_norm), 2.0));
        double eb = det_exp(dm_div(-dm_mul(b_norm, b_norm), 2.0));
        sh_yi = dm_div(dm_mul(dm_sub(ea, eb), is2pi), d_ii);
        sh_mii = m_ii;
      }
      sh_stop = y_stop;
      y_mii = m_ii;
    }
    if (im != i) {
      // :525-530, rows i <-> im over columns i0..n-1, then columns i <-> im,
      // in one pass: for k outside {i, im} the two swaps touch four distinct
      // elements; the 2 x 2 block on {i, im} ends up as (i,i) <- (im,im),
      // (im,im) <- (i,i), (i,im) <- (im,i), (im,i) <- (i,im)
      for (int64_t k = tid; k < n; k += blockDim.x) {
        if (k == i || k == im) {
          if (k == i) {
            const double ii = M[i * n + i], mm = M[im * n + im], im_i = M[i * n + im], i_im = M[im * n + i];
            M[i * n + i] = mm;
            M[im * n + im] = ii;
            M[im * n + i] = im_i;
            M[i * n + im] = i_im;
          }
          continue;
        }
        if (k >= i0) {
          const double t = M[k * n + i];
          M[k * n + i] = M[k * n + im];
          M[k * n + im] = t;
        }
        const double t = M[i * n + k];
        M[i * n + k] = M[im * n + k];
        M[im * n + k] = t;
      }
      __syncthreads();
    }
    if (yt && !y_stop) M[i * n + i] = y_mii;
    __syncthreads();
    if (sh_stop) {
      write_back();
      return;
    }
    const double m_ii = sh_mii, y_i = sh_yi;
    if (i == i0) {  // :547-554
      for (int64_t j = i + 1 + tid; j <= ii1; j += blockDim.x) {
        const int64_t q = j - i0;
        double m_ij = dm_div(M[j * n + i], m_ii);
        M[j * n + i] = m_ij;
        M[i * n + j] = m_ij;
        s_d[q] = dm_add(s_d[q], dm_mul(m_ij, m_ij));
        s_s[q] = dm_add(s_s[q], dm_mul(y_i, m_ij));
      }
    } else if (i < ii1) {  // :555-570
      for (int64_t j = i + 1 + tid; j <= ii1; j += blockDim.x) {
        const int64_t q = j - i0;
        // the ascending fma chain over l, its operands loaded 8 at a time
        // ahead of the chain
        double acc = 0.0;
        int64_t l = i0;
        for (; l + 8 <= i; l += 8) {
          double x[8], y[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            x[u] = M[(l + u) * n + j];
            y[u] = M[i * n + l + u];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = dm_fma(x[u], y[u], acc);
        }
        for (; l <= i - 1; ++l) acc = dm_fma(M[l * n + j], M[i * n + l], acc);
        double m_ij = dm_div(dm_sub(M[i * n + j], acc), m_ii);
        M[j * n + i] = m_ij;
        M[i * n + j] = m_ij;
        s_d[q] = dm_add(s_d[q], dm_mul(m_ij, m_ij));
        s_s[q] = dm_add(s_s[q], dm_mul(y_i, m_ij));
      }
    }
    __syncthreads();
  }
  write_back();
}

// One bs1 block of cholesky_genz! by a cluster of CTAs, 64 candidates each
// (panels of at most 512 candidates, blocks of at most 64 pivots).  One CTA
// for all candidates was bound by its FP64 pipe (two erf, two divisions and a
// square root a candidate and pivot) and by the row and column swaps, 4 n
// strided accesses of one SM a pivot: 10.7 us a pivot at 512 candidates with
// two finite bounds.  Here
//   * two threads a candidate take one bound each; det_erf's two polynomials
//     run as one chain with the coefficients picked from shared memory (the
//     shorter one led by zeros: the same bits), so lanes do not diverge;
//   * a candidate stays in its thread and only its position changes; M is read
//     where it lies (one coalesced column a pivot, in flight under the dot
//     products and the y_i) and permuted once per block by the whole GPU
//     (k_genz_gather, k_genz_scatter in chol.cu);
//   * each CTA sends its best candidate, factor entries included, to every CTA
//     of the cluster: one cluster barrier a pivot, after which every CTA takes
//     the pivot by itself.  The pivot's root and normalised bounds are its
//     score's (the same operands, the same bits), and a warp of its own forms
//     y_i under the others' dot products.
// Same operations in the same order as genz_block_dev: the same bits.
constexpr int kPivSlots = 64;     // candidates per CTA
constexpr int kPivThreads = 160;  // two per candidate, and the y_i warp
constexpr int kPivSlotThreads = 128;
constexpr int kPivCtas = 8;       // CTAs per cluster at most
constexpr int kPivMax = 64;       // pivots per block at most
constexpr int kPivPanel = kPivSlots * kPivCtas;

struct PivRec {
  unsigned long long key;  // argmin_key of the score, ~0: no candidate
  unsigned idx, pad;       // position << 16 | slot
  double m_raw, o, m_pp, nb, na;  // :533-541
  double f[kPivMax];
};
struct PivSmem {
  PivRec rec[2][kPivCtas];
  double f[kPivMax][kPivSlots];  // m[pivot, candidate]
  double o[kPivSlots], m[kPivSlots], r[kPivSlots], nb[kPivSlots], na[kPivSlots];
  double fd[kPivMax], y;
  double tab[2][29];
  unsigned long long wk[2][kPivSlotThreads / 32];
  unsigned wi[2][kPivSlotThreads / 32];
};
// What the block leaves for the permutation of M.
struct PivOut {
  int *ord;    // [panel] slot at each position
  double *f;   // [pivot][kPivPanel] factor entries by slot
  double *fd;  // [pivot] diagonal
  int *done;   // pivots completed (-1: the block did not run)
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int cta) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
  return r;
}
__device__ __forceinline__ void cluster_store(uint32_t a, unsigned long long v) {
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// det_erf with its coefficients in tab[0] (|x| < 2.5, padded to 29) and tab[1]
__device__ __forceinline__ double det_erf_tab(const double (*tab)[29], double x) {
  const double ax = fabs(x);
  const bool small = ax < 2.5;
  const double w = small ? dm_fma(dm_mul(ax, ax), 0x1.47ae147ae147bp-2, -1.0)
                         : dm_fma(ax, 0x1.2492492492492p-1, -0x1.36db6db6db6dbp+1);
  const double *c = tab[small ? 0 : 1];
  double q = c[28];
#pragma unroll
  for (int j = 27; j >= 0; --j) q = dm_fma(q, w, c[j]);
  double r = small ? dm_mul(ax, q) : dm_sub(1.0, q);
  r = ax < 6.0 ? r : 1.0;
  r = x < 0 ? -r : r;
  return x != x ? x : r;
}

__device__ __forceinline__ void genz_block_cluster(const double *M, int64_t n, double *a, double *b, double *dvec,
                                                   double *svec, int64_t *perm, int64_t i0, int64_t i1, int64_t ii1,
                                                   const double *eps0_ptr, int64_t *rank, PivOut out, PivSmem &sm) {
  const double c2 = dm_div(1.0, dm_sqrt(2.0));
  const double is2pi = dm_div(2.0, dm_sqrt(dm_mul(2.0, M_PI)));
  const double eps0 = eps0_ptr[0];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, C = (int)gridDim.x, cid = (int)blockIdx.x;
  const bool ywarp = tid >= kPivSlotThreads;
  const int sl = ywarp ? 0 : tid >> 1, slot = cid * kPivSlots + sl;
  const bool upper = (tid & 1) == 0;  // this thread's bound: b (even) or a (odd)
  const int len = (int)(ii1 - i0 + 1);
  const bool has = !ywarp && slot < len;
  const int64_t g = i0 + slot;
  if (rank[0] < n) {  // an earlier block already stopped
    if (cid == 0 && tid == 0) *out.done = -1;
    return;
  }
  if (tid < 58) {
    const double c_small[21] = DBGZ_ERF_SMALL_TABLE;
    const double c_mid[29] = DBGZ_ERFC_MID_TABLE;
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < 29; ++j) {
      if (tid == j && j < 21) v = c_small[j < 21 ? j : 0];
      if (tid == 29 + j) v = c_mid[j];
    }
    (&sm.tab[0][0])[tid] = v;
  }
  const double gd = has ? M[g * n + g] : 0.0, av = has ? a[g] : 0.0, bv = has ? b[g] : 0.0;
  const int64_t pv = has ? perm[g] : 0;
  const double xb = upper ? bv : av;
  double ds = 0.0, s = has ? svec[g] : 0.0;
  int pos = slot;
  const int np = (int)(i1 - i0 + 1);
  int done = np;
  cluster_sync_all();  // every CTA's shared memory is up (and this one's tables)
#pragma unroll 1
  for (int u = 0; u < np; ++u) {
    const int par = u & 1;
    // pivot scores (:500-512) and the CTA's least (argmin :514)
    unsigned long long key = ~0ull;
    unsigned idx = ~0u;
    if (!ywarp) {
      const double m_raw = dm_sub(gd, ds);
      const double m_kk = m_raw < 0 ? 0.0 : dm_sqrt(m_raw);
      const double nrm = dm_div(dm_sub(xb, s), m_kk);
      const double e = det_erf_tab(sm.tab, dm_mul(nrm, c2));
      const double eo = __shfl_xor_sync(0xffffffffu, e, 1);
      const double o = upper ? dm_sub(e, eo) : dm_sub(eo, e);
      if (upper) {
        sm.o[sl] = o;
        sm.m[sl] = m_raw;
        sm.r[sl] = m_kk;
        sm.nb[sl] = nrm;
        if (has && pos >= u) {
          key = argmin_key(o);
          idx = ((unsigned)pos << 16) | (unsigned)slot;
        }
      } else {
        sm.na[sl] = nrm;
      }
      warp_argmin(key, idx);
      if (lane == 0) {
        sm.wk[par][wid] = key;
        sm.wi[par][wid] = idx;
      }
    }
    __syncthreads();
    key = lane < kPivSlotThreads / 32 ? sm.wk[par][lane] : ~0ull;
    idx = lane < kPivSlotThreads / 32 ? sm.wi[par][lane] : ~0u;
    warp_argmin(key, idx);
    // this CTA's best candidate to every CTA (two buffers: a CTA that is a
    // step ahead writes the other one)
    {
      const int lb = key == ~0ull ? 0 : (int)(idx & 0xffffu) - cid * kPivSlots;
      const PivRec *R = &sm.rec[par][cid];
      const void *dst = nullptr;
      unsigned long long v = 0;
      if (tid < kPivMax) {
        if (tid < u) {
          dst = &R->f[tid];
          v = (unsigned long long)__double_as_longlong(sm.f[tid][lb]);
        }
      } else {
        switch (tid - kPivMax) {
          case 0: dst = &R->key; v = key; break;
          case 1: dst = &R->idx; v = idx; break;
          case 2: dst = &R->m_raw; v = (unsigned long long)__double_as_longlong(sm.m[lb]); break;
          case 3: dst = &R->o; v = (unsigned long long)__double_as_longlong(sm.o[lb]); break;
          case 4: dst = &R->m_pp; v = (unsigned long long)__double_as_longlong(sm.r[lb]); break;
          case 5: dst = &R->nb; v = (unsigned long long)__double_as_longlong(sm.nb[lb]); break;
          case 6: dst = &R->na; v = (unsigned long long)__double_as_longlong(sm.na[lb]); break;
          default: break;
        }
      }
      if (dst)
        for (int c = 0; c < C; ++c) cluster_store(cluster_addr(dst, c), v);
    }
    cluster_sync_all();
    key = lane < C ? sm.rec[par][lane].key : ~0ull;
    idx = lane < C ? sm.rec[par][lane].idx : ~0u;
    warp_argmin(key, idx);
    const int pslot = (int)(idx & 0xffffu), ppos = (int)(idx >> 16);
    const PivRec &R = sm.rec[par][pslot / kPivSlots];
    // :518-531: the pivot and the candidate at position u trade places
    if (slot == pslot) pos = u;
    else if (pos == u) pos = ppos;
    const bool live = has && pos > u;
    const double mij = live ? M[(i0 + pslot) * n + g] : 0.0;
    const double p_raw = R.m_raw;
    if (!(p_raw > eps0)) {  // the rank test of :533-537
      if (cid == 0 && tid == 0) rank[0] = i0 + u;
      done = u;
      break;
    }
    const double m_pp = R.m_pp;
    if (ywarp) {
      // y_i (:538-546), a side in half of the lanes (x / 2 = x * 0.5)
      const double nrm = upper ? R.nb : R.na;
      const double ex = det_exp(dm_mul(-dm_mul(nrm, nrm), 0.5));
      const double exo = __shfl_xor_sync(0xffffffffu, ex, 1);
      const double yi = dm_div(dm_mul(upper ? dm_sub(exo, ex) : dm_sub(ex, exo), is2pi), R.o);
      if (lane == 0) {
        sm.y = yi;
        sm.fd[u] = m_pp;
      }
      __syncwarp();
      asm volatile("bar.arrive 1, %0;" ::"n"(kPivThreads) : "memory");
      continue;
    }
    // the ascending fma chain over the block's pivots, eight loaded ahead
    double acc = 0.0, m = 0.0;
    int t = 0;
    if (u >= 8) {
      double x[8], y[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        x[q] = sm.f[q][sl];
        y[q] = R.f[q];
      }
      for (t = 8; t + 8 <= u; t += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          acc = dm_fma(x[q], y[q], acc);
          x[q] = sm.f[t + q][sl];
          y[q] = R.f[t + q];
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) acc = dm_fma(x[q], y[q], acc);
    }
    for (; t < u; ++t) acc = dm_fma(sm.f[t][sl], R.f[t], acc);
    if (live) {  // :547-570
      m = dm_div(dm_sub(mij, acc), m_pp);
      ds = dm_add(ds, dm_mul(m, m));
      if (upper) sm.f[u][sl] = m;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kPivThreads) : "memory");  // y_i is there
    if (live) s = dm_add(s, dm_mul(sm.y, m));
  }
  __syncthreads();
  if (has && upper) {
    const int64_t q = i0 + pos;
    dvec[q] = ds;
    svec[q] = s;
    a[q] = av;
    b[q] = bv;
    perm[q] = pv;
    out.ord[pos] = slot;
    for (int t = 0; t < done; ++t) out.f[t * kPivPanel + slot] = sm.f[t][sl];
  }
  if (cid == 0 && tid < done) out.fd[tid] = sm.fd[tid];
  if (cid == 0 && tid == 0) *out.done = done;
  cluster_sync_all();  // no CTA leaves while another may still write to it
}

// C[j,k] -= sum_{l=p0..p1} A(l,j) * B(l,k) for j,k in [c0, c1], one
// ascending fma chain per element.  A(l,j) = M[j,l] (row form, the
// reference's lower-triangle copy) when a_row, else M[l,j]; B(l,k) = M[l,k].
// One 32 x 32 output tile (j0, k0) per call, 256 threads (32 x 8).
constexpr int kTile = 32;
__device__ __forceinline__ void schur_tile_dev(double *M, int64_t n, int64_t p0, int64_t p1, int64_t c0,
                                               int64_t c1, int a_row, int64_t j0, int64_t k0) {
  __shared__ double As[kTile][kTile + 1];
  __shared__ double Bs[kTile][kTile + 1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t l0 = p0; l0 <= p1; l0 += kTile) {
    for (int r = ty; r < kTile; r += 8) {
      // As[l][c] = A(l0 + l, j0 + c); Bs[l][c] = B(l0 + l, k0 + c)
      int64_t l = l0 + tx, jj = j0 + r, kk = k0 + r;
      if (a_row) {
        int64_t lr = l0 + r, jc = j0 + tx;  // coalesced over j
        As[r][tx] = (lr <= p1 && jc <= c1) ? M[lr * n + jc] : 0.0;
      } else {
        As[tx][r] = (l <= p1 && jj <= c1) ? M[jj * n + l] : 0.0;
      }
      Bs[tx][r] = (l <= p1 && kk <= c1) ? M[kk * n + l] : 0.0;
    }
    __syncthreads();
    const int lmax = (int)((p1 - l0 + 1) < kTile ? (p1 - l0 + 1) : kTile);
    for (int l = 0; l < lmax; ++l) {
      double av = As[l][tx];
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r] = dm_fma(av, Bs[l][ty + 8 * r], acc[r]);
    }
    __syncthreads();
  }
  const int64_t j = j0 + tx;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    int64_t k = k0 + ty + 8 * r;
    if (j <= c1 && k <= c1) M[k * n + j] = dm_sub(M[k * n + j], acc[r]);
  }
}

}  // namespace cholk
