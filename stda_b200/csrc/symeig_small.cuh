// Lowest k eigenpairs of a small dense symmetric matrix (n <= kSymEigMaxN), for the
// Rayleigh-Ritz step of the Davidson solver and for dense windows, in four kernels
// with no host synchronisation:
//   1. k_symeig_tridiag: Householder reduction to tridiagonal form
//      T = Q^T A Q (LAPACK dsytd2, lower, restated) by one CTA or a cluster of
//      4 or 8, the matrix in registers (the scheme is described at the
//      kernel); d, e, tau and the reflectors go to a global workspace;
//   2. k_symeig_values (one CTA per eigenvalue): multisection on Sturm counts
//      (LAPACK dstebz's principle), each thread evaluating the count at one of
//      256 points of the current interval per round;
//   3. k_symeig_vectors (one warp per cluster of close eigenvalues, its work
//      arrays in shared memory): inverse iteration with a pivoted tridiagonal
//      LU (LAPACK dstein's scheme: shifts of equal eigenvalues nudged apart,
//      modified Gram-Schmidt against the earlier members of the cluster, two
//      iterations from a fixed start vector (bisection leaves the eigenvalue
//      within a few ulps of ||T||, so the first solve already grows the wanted
//      component by ~1/eps); the cluster threshold is
//      1e-5 ||T||, tighter than dstein's 1e-3, so that the dense Rayleigh-Ritz
//      spectra do not collapse into one serial cluster), vectors in T's basis;
//   4. k_symeig_backtransform (one CTA of 128 threads per eigenvector, held in
//      registers): z = Q y, the reflectors applied 8 at a time through the
//      triangular factors that phase 2 forms beside the eigenvalues.
// The vectors are orthogonal to 1e-15 ||A|| / gap (dense windows refine them).
// cuSOLVER's syevd takes 1-3 ms at n = 75-300, most of it launch and host
// synchronisation latency.
// Eigenvalues ascending in w[0..k), eigenvectors in the columns of Z (ld ldz).
// The *_b kernels run the same four phases for many problems per launch
// (blockIdx.y selects the problem; symeig_small_batched).
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace std2g {

constexpr int kTridiagThreads = 256;
constexpr int kSymEigMaxN = 320;       // 5 columns per warp in a cluster of 8 CTAs

constexpr int kBtBlock = 8;   // reflectors applied together by the back-transformation
__host__ __device__ inline int symeig_bt_blocks(int n) {
  return n > 2 ? (n - 2 + kBtBlock - 1) / kBtBlock : 0;
}

// global workspace (doubles): packed reflectors, d, e, tau, the triangular
// factors of the reflector blocks, and per eigenvector its y in T's basis (n)
__host__ __device__ inline size_t symeig_work_doubles(int n, int k) {
  return (size_t)n * (n + 1) / 2 + 3 * (size_t)n +
         (size_t)symeig_bt_blocks(n) * kBtBlock * kBtBlock + (size_t)k * n;
}

// packed lower column-major index of (i, j), i >= j
__device__ __forceinline__ int pk_idx(int i, int j, int n) {
  return j * (2 * n - j + 1) / 2 + (i - j);
}

// Number of eigenvalues below x of the scaled T: the sign changes of the
// leading principal minors p_i of T - x I,
//   p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1},
// with db[i] = {d_i, e_{i-1}^2}.  Dividing the recurrence by p_i gives the
// usual Sturm quotients, but puts an FP64 division on the serial chain; here
// the chain is one fused multiply-add per step.  |d - x| <= 2 and e^2 <= 1
// (scaled), so a step grows max(|p_i|, |p_{i-1}|) at most threefold, and e^2
// is kept >= kE2Min, so that 8 steps shrink it by at most 2^-800 and two
// consecutive minors never vanish: the pair is rescaled by a power of two
// every 8 steps.  A minor that is exactly zero counts once whatever the sign
// of the zero, since the next one then has the sign opposite to the last.
constexpr double kE2Min = 6.223015277861142e-61;   // 2^-200
__device__ __forceinline__ int sturm_count(const double2 *db, int n, double x) {
  double pm = 1.0, p = db[0].x - x;
  int neg = __double2hiint(p), cnt = (unsigned)neg >> 31;
  auto step = [&](double2 v) {
    const double t = fma(v.x - x, p, -(v.y * pm));
    pm = p;
    p = t;
    const int h = __double2hiint(t);
    cnt += (unsigned)(h ^ neg) >> 31;
    neg = h;
  };
  int i = 1;
  for (; i + 8 <= n; i += 8) {
    double2 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = db[i + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) step(v[u]);
    const int ex = max(__double2hiint(p) & 0x7fffffff, __double2hiint(pm) & 0x7fffffff) >> 20;
    const double sc = __hiloint2double(min(max(2046 - ex, 1), 2046) << 20, 0);
    p *= sc;
    pm *= sc;
  }
  for (; i < n; ++i) step(db[i]);
  return cnt;
}

// Gershgorin bounds of the rows i, i + stride, ... of T: interval [lo, hi] and
// largest absolute row sum nrm (reduced over the threads by the callers; min
// and max do not depend on the order)
__device__ __forceinline__ void tri_bounds(const double *d, const double *e, int n, int i0,
                                           int stride, double &lo, double &hi, double &nrm) {
  lo = 1e300;
  hi = -1e300;
  nrm = 0.0;
  for (int i = i0; i < n; i += stride) {
    const double ei = i + 1 < n ? fabs(e[i]) : 0.0, em = i > 0 ? fabs(e[i - 1]) : 0.0;
    lo = fmin(lo, d[i] - ei - em);
    hi = fmax(hi, d[i] + ei + em);
    nrm = fmax(nrm, fabs(d[i]) + ei + em);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
  }
}

struct SymEigWork {
  double *ap, *d, *e, *tau, *bt, *vec;
  __host__ __device__ SymEigWork(double *work, int n) {
    ap = work;
    d = ap + (size_t)n * (n + 1) / 2;
    e = d + n;
    tau = e + n;
    bt = tau + n;
    vec = bt + (size_t)symeig_bt_blocks(n) * kBtBlock * kBtBlock;
  }
};

// One problem of a batched launch (k_symeig_*_b: blockIdx.y selects the
// problem; every kernel of the batch covers the largest member, the blocks
// past a member's own size return early or stay idle as in a single launch).
struct SymEigJob {
  const double *A;
  int lda, n, k;
  double *w, *Z;
  int ldz;
  double *work;
  int *info;
};

// ---- 1. tridiagonal reduction (Q^T A Q = T, Q = H_0 ... H_{n-3}) ----------
// Latency-bound: n - 2 dependent steps.  The matrix stays in the registers of
// 8 C warps (C CTAs of one cluster): warp g holds the whole columns
// j = g, g + 8 C, ... (CPW of them), lane l the rows l, l + 32, ... (RB of
// them).  Every warp keeps itself informed instead of waiting for a block-wide
// reduction: each one forms the reflector of the current column (cur, in
// shared memory) and later p^T v with its own shuffles, all with the same
// arithmetic, so a step takes two barriers:
//   v, tau from cur; p_j = tau (A v)_j for the own columns, written to the p
//   array of every CTA; the owner of column c+1 publishes it;
//   cluster barrier;
//   w = p - (tau p^T v / 2) v; thread i updates element i of column c+1 into
//   the next cur; A -= v w^T + w v^T on the own columns;
//   CTA barrier.
// The steps run in phases of 32, so that the row blocks and columns that are
// done drop out at compile time; eight warps, not more, because each repeats
// the square root and the divisions of the reflector.
// p and the published column alternate between two buffers: a CTA that writes
// buffer (c+1) % 2 has passed the cluster barrier of step c, which every CTA
// enters only after reading that buffer in step c-1.
// Measured for the whole eigensolve (n = 100 / 300, 25 / 62 pairs): 347 -> 220 us
// and 1422 -> 799 us against columns in shared memory with block-wide reductions
// and 4 / 8 CTAs.
template <int C_, int RB_, int CPW_>
struct TridiagShape {
  static constexpr int C = C_, RB = RB_, CPW = CPW_;
};
constexpr int kTridiagWarps = kTridiagThreads / 32;

template <int I, int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

// Sums of NQ values over the warp: on return lane l holds in x[0] the sum of
// value q(l), the top log2 bits of the lane (NQ rounded up to a power of two):
// the halves of the lanes exchange halves of the values, NQ - 1 shuffles
// instead of 5 NQ, then the rest reduce one value.
template <int NQ>
__device__ __forceinline__ int warp_sums(double (&x)[NQ], int lane) {
  constexpr int P = NQ <= 1 ? 1 : NQ <= 2 ? 2 : NQ <= 4 ? 4 : NQ <= 8 ? 8 : 16;
  double y[P];
#pragma unroll
  for (int q = 0; q < P; ++q) y[q] = q < NQ ? x[q] : 0.0;
  int o = 16, q0 = 0;
#pragma unroll
  for (int h = P / 2; h > 0; h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const double send = up ? y[q] : y[q + h], keep = up ? y[q + h] : y[q];
      y[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    q0 += up ? h : 0;
    o >>= 1;
  }
#pragma unroll
  for (int b = 16; b > 0; b >>= 1)
    if (b <= o) y[0] += __shfl_xor_sync(0xffffffffu, y[0], b);
  x[0] = y[0];
  return q0;
}

// x, or 0 below 2^-485 (1e-146): the squares of what is left are exact to more than 53
// bits.  (A column of entries about 1e-159 had squares of a few bits, and its
// reflector was not orthogonal.)  A test of the column's norm instead, with a reflector
// formed from scaled entries behind it, made the reduction 4 % slower.
__device__ __forceinline__ double symeig_keep(double x) {
  return (__double2hiint(x) & 0x7fffffff) < (1023 - 485) << 20 ? 0.0 : x;
}

template <class Shape>
__device__ __forceinline__ void
symeig_tridiag_body(const double *__restrict__ A, int lda, int n, double *__restrict__ work) {
  constexpr int C = Shape::C, RB = Shape::RB, CPW = Shape::CPW, LD = 32 * RB;
  constexpr int G = kTridiagWarps * C;
  namespace cg = cooperative_groups;
  __shared__ double s_cur[2][LD], s_p[2][LD], s_col[2][LD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int rank = 0;
  if constexpr (C > 1) rank = (int)cg::this_cluster().block_rank();
  const int gw = rank * kTridiagWarps + warp;   // columns gw + G q
  const SymEigWork g(work, n);
  double a[CPW][RB];
#pragma unroll
  for (int q = 0; q < CPW; ++q)
#pragma unroll
    for (int t = 0; t < RB; ++t) {
      const int j = gw + G * q, i = lane + 32 * t;
      a[q][t] = i < n && j < n ? A[max(i, j) + (size_t)lda * min(i, j)] : 0.0;
    }
  for (int i = tid; i < LD; i += kTridiagThreads) {
    s_cur[0][i] = i < n ? symeig_keep(A[i]) : 0.0;   // column 0
    s_cur[1][i] = 0.0;
    s_p[0][i] = s_p[1][i] = 0.0;
    s_col[0][i] = s_col[1][i] = 0.0;
  }
  if constexpr (C > 1) cg::this_cluster().sync();   // buffers cleared before remote writes
  else __syncthreads();
  static_for<0, RB>([&](auto phase) {
    constexpr int T0 = decltype(phase)::value, NT = RB - T0;
    constexpr int Q0 = 32 * T0 / G, NQ = CPW - Q0;   // columns below G Q0 are done
    for (int c = max(0, 32 * T0 - 1); c < min(n - 2, 32 * T0 + 31); ++c) {
      const int r0 = c + 1, buf = c & 1, l0 = lane + 32 * T0;
      const double *cur = s_cur[buf];
      // ---- reflector H_c = I - tau v v^T of rows r0..n-1 of cur (LAPACK
      // dlarfg's convention: v[r0] = 1, beta = -sign(alpha) ||x||)
      double v[NT], xn2 = 0.0;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        v[t] = l0 + 32 * t > r0 ? cur[l0 + 32 * t] : 0.0;
        xn2 = fma(v[t], v[t], xn2);
      }
      const double alpha = cur[r0];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, o);
      double tc = 0.0, beta = alpha, scal = 0.0;
      if (xn2 != 0.0) {
        beta = -copysign(sqrt(fma(alpha, alpha, xn2)), alpha);
        tc = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) v[t] = l0 + 32 * t == r0 ? 1.0 : v[t] * scal;
      if (gw == 0) {   // kept for the back-transformation
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int i = l0 + 32 * t;
          if (i > r0 && i < n) g.ap[pk_idx(i, c, n)] = v[t];
        }
        if (lane == 0) {
          g.tau[c] = tc;
          g.e[c] = beta;
          g.d[c] = cur[c];
        }
      }
      // ---- p_j = tau (A v)_j, and column c+1 published by its owner
      double ps[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double s = 0.0;
#pragma unroll
        for (int t = 0; t < NT; ++t) s = fma(a[Q0 + q][T0 + t], v[t], s);
        ps[q] = s;
        if (gw + G * (Q0 + q) == r0)
#pragma unroll
          for (int t = 0; t < NT; ++t) s_col[buf][l0 + 32 * t] = a[Q0 + q][T0 + t];
      }
      const int qs = warp_sums(ps, lane);
      {
        // the lanes of one value q write it, lane (their index) mod C to CTA .. C
        constexpr int P = NQ <= 1 ? 1 : NQ <= 2 ? 2 : NQ <= 4 ? 4 : NQ <= 8 ? 8 : 16;
        constexpr int L = 32 / P;   // lanes holding the same sum
        const int j = gw + G * (Q0 + qs);
        if (qs < NQ && j >= r0 && j < n) {
#pragma unroll
          for (int k = 0; k < (C + L - 1) / L; ++k) {
            const int to = lane % L + L * k;
            if (to < C) {
              if constexpr (C > 1) cg::this_cluster().map_shared_rank(s_p[buf], to)[j] = tc * ps[0];
              else s_p[buf][j] = tc * ps[0];
            }
          }
        }
      }
      const double *rc = s_col[buf];
      if constexpr (C > 1) {
        cg::this_cluster().sync();
        rc = cg::this_cluster().map_shared_rank(s_col[buf], (r0 % G) / kTridiagWarps);
      } else {
        __syncthreads();
      }
      // ---- w = p - K v, the next column, the rank-2 update
      constexpr int NE = (LD + kTridiagThreads - 1) / kTridiagThreads;
      double rci[NE];
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int i = tid + kTridiagThreads * k;
        rci[k] = i >= r0 && i < n ? rc[i] : 0.0;
      }
      const double *p = s_p[buf];
      double w[NT], pv = 0.0;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        w[t] = l0 + 32 * t >= r0 ? p[l0 + 32 * t] : 0.0;
        pv = fma(w[t], v[t], pv);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pv += __shfl_xor_sync(0xffffffffu, pv, o);
      const double K = 0.5 * tc * pv;
#pragma unroll
      for (int k = 0; k < NE; ++k) {   // element i of column r0; v[r0] = 1
        const int i = tid + kTridiagThreads * k;
        if (i >= r0 && i < n) {
          const double vi = i == r0 ? 1.0 : cur[i] * scal;
          s_cur[buf ^ 1][i] = symeig_keep(rci[k] - fma(vi, p[r0] - K, p[i] - K * vi));
        }
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) w[t] = fma(-K, v[t], w[t]);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int j = gw + G * (Q0 + q);
        // columns that are done take a zero update
        const double vj = j > r0 && j < n ? cur[j] * scal : 0.0;
        const double wj = j > r0 && j < n ? fma(-K, vj, p[j]) : 0.0;
#pragma unroll
        for (int t = 0; t < NT; ++t)
          a[Q0 + q][T0 + t] = fma(-v[t], wj, fma(-w[t], vj, a[Q0 + q][T0 + t]));
      }
      __syncthreads();
    }
  });
  // the trailing 2 x 2 block: cur holds column n-2, column n-1 is on its owner
  const double *cur = s_cur[max(n - 2, 0) & 1];
  if (gw == 0 && lane == 0 && n >= 2) {
    g.d[n - 2] = cur[n - 2];
    g.e[n - 2] = cur[n - 1];
    g.tau[n - 2] = 0.0;
  }
  if (gw == (n - 1) % G && lane == (n - 1) % 32) {
#pragma unroll
    for (int q = 0; q < CPW; ++q)
#pragma unroll
      for (int t = 0; t < RB; ++t)
        if (gw + G * q == n - 1 && lane + 32 * t == n - 1) g.d[n - 1] = a[q][t];
    g.e[n - 1] = 0.0;
    g.tau[n - 1] = 0.0;
  }
  if constexpr (C > 1) cg::this_cluster().sync();   // shared memory still read by other CTAs
}

template <class Shape>
__global__ void __launch_bounds__(kTridiagThreads, 1)
k_symeig_tridiag(const double *__restrict__ A, int lda, int n, double *__restrict__ work) {
  symeig_tridiag_body<Shape>(A, lda, n, work);
}

// batched form: cluster blockIdx.y solves jobs[blockIdx.y]
template <class Shape>
__global__ void __launch_bounds__(kTridiagThreads, 1)
k_symeig_tridiag_b(const SymEigJob *__restrict__ jobs) {
  const SymEigJob j = jobs[blockIdx.y];
  symeig_tridiag_body<Shape>(j.A, j.lda, j.n, j.work);
}

// f(shape index, Shape) for the shape that serves size n: the fewest CTAs whose
// registers hold the matrix, up to where more of them were faster (whole
// eigensolve: n = 96 188 us with one CTA, 212 / 203 with 2 / 4; n = 128 275
// against 295 / 279; n = 150 343 with 4 against 372 / 342 with 2 / 8; n = 192
// 439 with 8 against 453 / 500 with 4 / 2; n = 256 652 with 8 against 684)
constexpr int kTridiagShapes = 8;
template <class F>
inline void symeig_tridiag_shape(int n, F &&f) {
  if (n <= 32) f(0, TridiagShape<1, 1, 4>{});
  else if (n <= 64) f(1, TridiagShape<1, 2, 8>{});
  else if (n <= 96) f(2, TridiagShape<1, 3, 12>{});
  else if (n <= 128) f(3, TridiagShape<1, 4, 16>{});
  else if (n <= 160) f(4, TridiagShape<4, 5, 5>{});
  else if (n <= 192) f(5, TridiagShape<8, 6, 3>{});
  else if (n <= 256) f(6, TridiagShape<8, 8, 4>{});
  else f(7, TridiagShape<8, 10, 5>{});
}

// ---- 2. eigenvalues: multisection on Sturm counts, one CTA per eigenvalue ---
// A round evaluates the count at kValThreads points of the interval, so that
// it shrinks 257-fold: 7 rounds instead of the 11 of one warp's 32 points.
// Measured for the whole eigensolve (25 / 62 pairs of n = 100 / 300): 457 -> 371 us and
// 1744 -> 1492 us against one warp per eigenvalue with the quotient recurrence.
constexpr int kSymEigWarps = 8;   // warps per CTA of phase 3
constexpr int kValThreads = 256;

__host__ __device__ inline size_t symeig_val_smem_bytes(int n) {
  return sizeof(double) * (size_t)n * kBtBlock;   // values: 4 n, block factors: 8 n
}

__device__ __forceinline__ void
symeig_values_body(int j, int n, const double *__restrict__ work, double *__restrict__ w) {
  extern __shared__ __align__(16) double sm[];
  double2 *db = (double2 *)sm;                 // scaled {d_i, e_{i-1}^2}
  double *d = sm + 2 * (size_t)n, *e = d + n;
  __shared__ double red[3][kValThreads / 32];
  __shared__ int first[2][kValThreads / 32];
  const SymEigWork g(const_cast<double *>(work), n);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < n; i += kValThreads) {
    d[i] = g.d[i];
    e[i] = g.e[i];
  }
  __syncthreads();
  double a, b, nrm;
  tri_bounds(d, e, n, tid, kValThreads, a, b, nrm);
  if (lane == 0) {
    red[0][warp] = a;
    red[1][warp] = b;
    red[2][warp] = nrm;
  }
  __syncthreads();
  for (int q = 0; q < kValThreads / 32; ++q) {
    a = fmin(a, red[0][q]);
    b = fmax(b, red[1][q]);
    nrm = fmax(nrm, red[2][q]);
  }
  // scale by a power of two to ||T|| in [1/2, 1) (exact)
  int ex = 0;
  if (nrm > 0.0 && nrm < 1e300) frexp(nrm, &ex);
  const double sc = ldexp(1.0, -ex), eps = 2.220446049250313e-16;
  a = a * sc - (2.0 * eps * nrm * sc + 1e-300);
  b = b * sc + (2.0 * eps * nrm * sc + 1e-300);
  for (int i = tid; i < n; i += kValThreads) {
    const double em = i > 0 ? e[i - 1] * sc : 0.0;
    db[i] = make_double2(d[i] * sc, fmax(em * em, kE2Min));
  }
  __syncthreads();
  for (int round = 0; round < 64; ++round) {
    if (b - a <= 2.0 * eps * fmax(fabs(a), fabs(b)) + 1e-300) break;
    const double h = (b - a) * (1.0 / (kValThreads + 1));
    const int cnt = sturm_count(db, n, fma(h, (double)(tid + 1), a));
    // the first point with more than j eigenvalues below it bounds eigenvalue j
    const unsigned above = __ballot_sync(0xffffffffu, cnt > j);
    if (lane == 0) first[round & 1][warp] = above ? __ffs(above) - 1 : 32;
    __syncthreads();
    int l = kValThreads;
    for (int q = kValThreads / 32 - 1; q >= 0; --q) {
      const int f = first[round & 1][q];
      if (f < 32) l = 32 * q + f;
    }
    const double na = l == 0 ? a : fma(h, (double)l, a);
    const double nb = l == kValThreads ? b : fma(h, (double)(l + 1), a);
    a = na;
    b = nb;
  }
  if (tid == 0) w[j] = ldexp(0.5 * (a + b), ex);
}

// entry i of the reflector vector of H_c (0 for i <= c, 1 at c + 1)
__device__ __forceinline__ double symeig_v(const SymEigWork &g, int i, int c, int n) {
  return c < 0 || i <= c ? 0.0 : (i == c + 1 ? 1.0 : g.ap[pk_idx(i, c, n)]);
}

// Triangular factor of reflector block b (for phase 4), formed beside the
// eigenvalues on CTAs that would otherwise idle: the block applies H_c,
// c = n-3-8b-r, in the order r = 0 .. 7, i.e. y <- y - sum_r f_r v_r with
// f_r = tau_r (v_r^T y - sum_{q<r} (v_r^T v_q) f_q), so f = F V^T y with
//   F_rr = tau_r,  F_rq = -tau_r sum_{q<=s<r} (v_r^T v_s) F_sq.
__device__ __forceinline__ void symeig_block_factor(int b, int n, double *__restrict__ work) {
  extern __shared__ __align__(16) double sm[];   // V[kBtBlock][n]
  __shared__ double gram[kBtBlock][kBtBlock];
  const SymEigWork g(work, n);
  const int c1 = n - 3 - kBtBlock * b, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int x = threadIdx.x; x < kBtBlock * n; x += kValThreads)
    sm[x] = symeig_v(g, x % n, c1 - x / n, n);
  __syncthreads();
  for (int x = warp; x < kBtBlock * kBtBlock; x += kValThreads / 32) {
    const int r = x / kBtBlock, q = x % kBtBlock;
    if (q >= r) continue;
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += sm[r * n + i] * sm[q * n + i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) gram[r][q] = s;
  }
  __syncthreads();
  if (threadIdx.x < kBtBlock) {
    const int q = threadIdx.x;
    double f[kBtBlock];
#pragma unroll
    for (int r = 0; r < kBtBlock; ++r) {
      const double t = c1 - r >= 0 ? g.tau[c1 - r] : 0.0;
      double s = 0.0;
#pragma unroll
      for (int u = 0; u < r; ++u) s += u >= q ? gram[r][u] * f[u] : 0.0;
      f[r] = r < q ? 0.0 : (r == q ? t : -t * s);
      g.bt[((size_t)b * kBtBlock + r) * kBtBlock + q] = f[r];
    }
  }
}

// blocks 0 .. k-1: one eigenvalue each; block k + b: reflector block b
__global__ void __launch_bounds__(kValThreads)
k_symeig_values(int n, int k, double *__restrict__ work, double *__restrict__ w) {
  if (blockIdx.x < k) symeig_values_body(blockIdx.x, n, work, w);
  else symeig_block_factor(blockIdx.x - k, n, work);
}

__global__ void __launch_bounds__(kValThreads)
k_symeig_values_b(const SymEigJob *__restrict__ jobs) {
  const SymEigJob j = jobs[blockIdx.y];
  if (blockIdx.x < j.k) symeig_values_body(blockIdx.x, j.n, j.work, j.w);
  else if (blockIdx.x - j.k < symeig_bt_blocks(j.n))
    symeig_block_factor(blockIdx.x - j.k, j.n, j.work);
}

// ---- 3. eigenvectors of T, one warp per cluster of close eigenvalues --------
// Cluster threshold: eigenvalues closer than 1e-5 ||T|| are orthogonalised
// against each other; further apart, inverse iteration alone gives vectors
// orthogonal to ~eps ||T|| / gap <= 2e-11.  The factorisation and the solves
// are serial chains in one lane, so they are arranged to carry as little as
// possible: one reciprocal per row in the factorisation, rows of U divided by
// their pivots beforehand by all lanes (one multiply-add per row in the back
// substitution), the running values in registers, the rows' other entries
// loaded four at a time; the first solve starts at the back substitution (its
// start vector stands for L^-1 P y).  Whole eigensolve: -25 us at n = 100,
// -70 us at n = 300 against the plain chains.
// Shared memory: d, e, then per warp y, 1 / pivot, {u1, u2} (the two
// super-diagonals of U over the pivot), {multiplier, row-swap flag}.
__host__ __device__ inline size_t symeig_vec_smem_bytes(int n) {
  const size_t np = (size_t)(n + 1) & ~(size_t)1;   // 16-byte rows
  return sizeof(double) * (2 * np + (size_t)kSymEigWarps * 6 * np);
}

// Entry i of member m's start vector: +-[1/2, 1), from a hash of (i, m) that mixes
// the two through products.  The start vectors of a cluster of equal eigenvalues have
// to be independent of each other, since the Gram-Schmidt steps keep only what is new
// in each: exclusive-or and shifts of one function of i and one of m span 17
// directions, and a 150-fold eigenvalue of 2 x 2 blocks got dependent vectors.
__device__ __forceinline__ double symeig_start(int i, int m) {
  unsigned h = (unsigned)(i + 1) * 0x9E3779B1u + (unsigned)(m + 1) * 0x85EBCA77u;
  h = (h ^ h >> 16) * 0x9E3779B1u;
  h = (h ^ h >> 15) * 0x85EBCA77u;
  h ^= h >> 16;
  const double v = 0.5 + (double)(h >> 1) * 0x1p-32;
  return h & 1 ? v : -v;
}

__device__ __forceinline__ void
symeig_vectors_body(int n, int k, double *__restrict__ work, const double *__restrict__ w) {
  extern __shared__ __align__(16) double sm[];
  const int np = (n + 1) & ~1;
  double *d = sm, *e = sm + np;
  const SymEigWork g(work, n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] = g.d[i];
    e[i] = g.e[i];   // e[n-1] = 0
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int j0 = blockIdx.x * kSymEigWarps + wl;
  if (j0 >= k) return;
  const double eps = 2.220446049250313e-16;
  double lo_, hi_, nrm;
  tri_bounds(d, e, n, lane, 32, lo_, hi_, nrm);
  const double ortol = 1e-5 * nrm, pertol = 10.0 * eps * nrm, tiny = eps * nrm + 1e-300;
  if (j0 > 0 && (w[j0] - w[j0 - 1]) <= ortol) return;   // not the first of its cluster
  int j1 = j0 + 1;
  while (j1 < k && (w[j1] - w[j1 - 1]) <= ortol) ++j1;
  double *y = sm + 2 * np + (size_t)wl * 6 * np, *ua = y + np;
  double2 *ub = (double2 *)(ua + np), *mf = ub + np;
  double lam_prev = 0.0;
  for (int m = j0; m < j1; ++m) {
    double lam = w[m];
    if (m > j0 && lam - lam_prev < pertol) lam = lam_prev + pertol;
    lam_prev = lam;
    if (lane == 0) {   // T - lam I = P L U with partial pivoting
      double a0 = d[0] - lam, b0 = e[0];
      for (int i = 0; i + 1 < n; ++i) {
        const double sub = e[i], dn = d[i + 1] - lam, en = e[i + 1];
        const bool sw = fabs(a0) < fabs(sub);   // swap rows i and i+1
        double piv = sw ? sub : a0;
        if (fabs(piv) < tiny) piv = piv < 0.0 ? -tiny : tiny;
        const double inv = 1.0 / piv, ml = (sw ? a0 : sub) * inv;
        const double u1 = sw ? dn : b0, u2 = sw ? en : 0.0;
        ua[i] = inv;
        ub[i] = make_double2(u1, u2);
        mf[i] = make_double2(ml, sw ? 1.0 : 0.0);
        a0 = fma(-ml, u1, sw ? b0 : dn);
        b0 = sw ? -ml * en : en;
      }
      double piv = a0;
      if (fabs(piv) < tiny) piv = piv < 0.0 ? -tiny : tiny;
      ua[n - 1] = 1.0 / piv;
      ub[n - 1] = make_double2(0.0, 0.0);
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
      const double ia = ua[i];
      const double2 u = ub[i];
      ub[i] = make_double2(-u.x * ia, -u.y * ia);
      y[i] = symeig_start(i, m) * ia;
    }
    __syncwarp();
    for (int it = 0; it < 2; ++it) {
      if (lane == 0) {
        if (it > 0) {   // y <- L^-1 P y, each row over its pivot
          double c = y[0];
          int i = 0;
          for (; i + 4 < n; i += 4) {
            double yn[4], ia[4];
            double2 f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              yn[u] = y[i + 1 + u];
              f[u] = mf[i + u];
              ia[u] = ua[i + u];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const bool sw = f[u].y != 0.0;
              const double top = sw ? yn[u] : c, bot = sw ? c : yn[u];
              y[i + u] = top * ia[u];
              c = fma(-f[u].x, top, bot);
            }
          }
          for (; i + 1 < n; ++i) {
            const double yn = y[i + 1];
            const bool sw = mf[i].y != 0.0;
            const double top = sw ? yn : c, bot = sw ? c : yn;
            y[i] = top * ua[i];
            c = fma(-mf[i].x, top, bot);
          }
          y[n - 1] = c * ua[n - 1];
        }
        double x1 = 0.0, x2 = 0.0;   // U x = y
        int i = n - 1;
        for (; i >= 3; i -= 4) {
          double yv[4];
          double2 f[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            yv[u] = y[i - u];
            f[u] = ub[i - u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double x = fma(f[u].x, x1, fma(f[u].y, x2, yv[u]));
            y[i - u] = x;
            x2 = x1;
            x1 = x;
          }
        }
        for (; i >= 0; --i) {
          const double x = fma(ub[i].x, x1, fma(ub[i].y, x2, y[i]));
          y[i] = x;
          x2 = x1;
          x1 = x;
        }
      }
      __syncwarp();
      for (int q = j0; q < m; ++q) {   // MGS against earlier cluster members (in T's basis)
        const double *zq = g.vec + (size_t)q * n;
        double dot = 0.0;
        for (int i = lane; i < n; i += 32) dot += zq[i] * y[i];
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        for (int i = lane; i < n; i += 32) y[i] -= dot * zq[i];
        __syncwarp();
      }
      double nn = 0.0;
      for (int i = lane; i < n; i += 32) nn += y[i] * y[i];
      for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
      const double inv = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
      for (int i = lane; i < n; i += 32) y[i] *= inv;
      __syncwarp();
    }
    // the member's vector in T's basis, for the MGS of the later members
    for (int i = lane; i < n; i += 32) g.vec[(size_t)m * n + i] = y[i];
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kSymEigWarps * 32)
k_symeig_vectors(int n, int k, double *__restrict__ work, const double *__restrict__ w) {
  symeig_vectors_body(n, k, work, w);
}

__global__ void __launch_bounds__(kSymEigWarps * 32)
k_symeig_vectors_b(const SymEigJob *__restrict__ jobs) {
  const SymEigJob j = jobs[blockIdx.y];
  symeig_vectors_body(j.n, j.k, j.work, j.w);
}

// ---- 4. back-transformation z = H_0 ... H_{n-3} y ----------------------------
// One CTA of 128 threads per eigenvector, thread = row mod 128 (RL rows each),
// the vector in registers.  The reflectors come in blocks of 8: the 8 dot
// products v_r^T y are independent, the coefficients follow through the
// block's triangular factor (symeig_block_factor), and the next block is
// loaded meanwhile, so a block costs one reduction and one barrier where
// reflector after reflector cost eight reductions.  Whole eigensolve: 220 -> 189 us
// at n = 100, 799 -> 656 us at n = 300 against one warp per vector with the
// reflectors in shared memory.
constexpr int kBtThreads = 128;
template <int RL>
__device__ __forceinline__ void
symeig_backtransform_rows(int m, int n, const double *__restrict__ work,
                          const double *__restrict__ w, double *__restrict__ Z, int ldz,
                          int *info) {
  constexpr int B = kBtBlock, NW = kBtThreads / 32;
  __shared__ double part[2][NW][B];
  const SymEigWork g(const_cast<double *>(work), n);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double y[RL], v[B][RL], nx[B][RL];
#pragma unroll
  for (int t = 0; t < RL; ++t) {
    const int i = tid + kBtThreads * t;
    y[t] = i < n ? g.vec[(size_t)m * n + i] : 0.0;
  }
  const int nb = symeig_bt_blocks(n);
  double frow[B], fnx[B];   // row lane % B of the block's factor
  auto load = [&](int b, double (&x)[B][RL], double (&f)[B]) {
    const int c1 = n - 3 - B * b;
#pragma unroll
    for (int r = 0; r < B; ++r) {
#pragma unroll
      for (int t = 0; t < RL; ++t) {
        const int i = tid + kBtThreads * t;
        x[r][t] = i < n ? symeig_v(g, i, c1 - r, n) : 0.0;
      }
      f[r] = g.bt[((size_t)b * B + lane % B) * B + r];
    }
  };
  if (nb > 0) load(0, nx, fnx);
  for (int b = 0; b < nb; ++b) {
#pragma unroll
    for (int r = 0; r < B; ++r) {
      frow[r] = fnx[r];
#pragma unroll
      for (int t = 0; t < RL; ++t) v[r][t] = nx[r][t];
    }
    if (b + 1 < nb) load(b + 1, nx, fnx);
    double s[B];
#pragma unroll
    for (int r = 0; r < B; ++r) {
      s[r] = 0.0;
#pragma unroll
      for (int t = 0; t < RL; ++t) s[r] = fma(v[r][t], y[t], s[r]);
    }
    const int q = warp_sums(s, lane);
    if (lane % (32 / B) == 0) part[b & 1][warp][q] = s[0];
    __syncthreads();
    double dot = 0.0, f = 0.0;   // dot product lane % B, coefficient lane % B
#pragma unroll
    for (int u = 0; u < NW; ++u) dot += part[b & 1][u][lane % B];
#pragma unroll
    for (int r = 0; r < B; ++r) f = fma(frow[r], __shfl_sync(0xffffffffu, dot, r), f);
#pragma unroll
    for (int r = 0; r < B; ++r) {
      const double fr = __shfl_sync(0xffffffffu, f, r);
#pragma unroll
      for (int t = 0; t < RL; ++t) y[t] = fma(-fr, v[r][t], y[t]);
    }
  }
  bool bad = !isfinite(w[m]);
#pragma unroll
  for (int t = 0; t < RL; ++t) {
    const int i = tid + kBtThreads * t;
    if (i < n) {
      bad |= !isfinite(y[t]);
      Z[i + (size_t)ldz * m] = y[t];
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(info, 1);
}

__device__ __forceinline__ void
symeig_backtransform_body(int m, int n, const double *__restrict__ work,
                          const double *__restrict__ w, double *__restrict__ Z, int ldz,
                          int *info) {
  if (n <= kBtThreads) symeig_backtransform_rows<1>(m, n, work, w, Z, ldz, info);
  else if (n <= 2 * kBtThreads) symeig_backtransform_rows<2>(m, n, work, w, Z, ldz, info);
  else symeig_backtransform_rows<3>(m, n, work, w, Z, ldz, info);
}
static_assert(kSymEigMaxN <= 3 * kBtThreads, "rows per thread");

__global__ void __launch_bounds__(kBtThreads)
k_symeig_backtransform(int n, const double *__restrict__ work, const double *__restrict__ w,
                       double *__restrict__ Z, int ldz, int *info) {
  symeig_backtransform_body(blockIdx.x, n, work, w, Z, ldz, info);
}

__global__ void __launch_bounds__(kBtThreads)
k_symeig_backtransform_b(const SymEigJob *__restrict__ jobs) {
  const SymEigJob j = jobs[blockIdx.y];
  if (blockIdx.x < j.k) symeig_backtransform_body(blockIdx.x, j.n, j.work, j.w, j.Z, j.ldz, j.info);
}

// host launchers: n <= kSymEigMaxN, k <= n; work: symeig_work_doubles(n, k).
// Phases 1 and 2 (the lowest k eigenvalues), then 3 and 4 (vectors of the lowest k).
inline void symeig_small_values(cudaStream_t s, const double *A, int lda, int n, int k, double *w,
                                double *work) {
  if (n < 1 || n > kSymEigMaxN || k < 1 || k > n)
    throw Error{STD2G_EINVAL, "symeig_small: size out of range"};
  symeig_tridiag_shape(n, [&](int, auto shape) {
    using Shape = decltype(shape);
    launch_cluster(k_symeig_tridiag<Shape>, dim3(Shape::C), kTridiagThreads, 0, dim3(Shape::C), s,
                   A, lda, n, work);
  });
  S2G_LAUNCH(k_symeig_values, k + symeig_bt_blocks(n), kValThreads, symeig_val_smem_bytes(n), s, n,
             k, work, w);
}

inline void symeig_small_vectors(cudaStream_t s, int n, int k, const double *w, double *Z, int ldz,
                                 double *work, int *info) {
  // the attribute is the same for every call (contexts on other host threads
  // launch the same kernel concurrently), the launch takes what n needs
  S2G_CUDA(cudaFuncSetAttribute(k_symeig_vectors, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)symeig_vec_smem_bytes(kSymEigMaxN)));
  const int nb = (k + kSymEigWarps - 1) / kSymEigWarps;
  S2G_LAUNCH(k_symeig_vectors, nb, kSymEigWarps * 32, symeig_vec_smem_bytes(n), s, n, k, work, w);
  S2G_LAUNCH(k_symeig_backtransform, k, kBtThreads, 0, s, n, work, w, Z, ldz, info);
}

inline void symeig_small(cudaStream_t s, const double *A, int lda, int n, int k, double *w,
                         double *Z, int ldz, double *work, int *info) {
  symeig_small_values(s, A, lda, n, k, w, work);
  symeig_small_vectors(s, n, k, w, Z, ldz, work, info);
}

// Batched launcher: the problems of `jobs` (each n <= kSymEigMaxN, 1 <= k <= n)
// in three launches for all of them, plus one tridiagonalisation launch per
// shape (symeig_tridiag_shape).  The job table goes to `dj` (same stream: a later upload
// waits for these kernels), from `stage` when given.
inline void symeig_small_batched(cudaStream_t s, const std::vector<SymEigJob> &jobs,
                                 DBuf<SymEigJob> &dj, PinnedArena *stage = nullptr) {
  if (jobs.empty()) return;
  std::vector<SymEigJob> ord;
  int count[kTridiagShapes] = {0}, nmax = 0, kmax = 0;
  for (int shape = 0; shape < kTridiagShapes; ++shape)
    for (const SymEigJob &j : jobs) {
      if (j.n < 1 || j.n > kSymEigMaxN || j.k < 1 || j.k > j.n)
        throw Error{STD2G_EINVAL, "symeig_small_batched: size out of range"};
      int mine = 0;
      symeig_tridiag_shape(j.n, [&](int q, auto) { mine = q; });
      if (mine != shape) continue;
      ord.push_back(j);
      ++count[shape];
      nmax = std::max(nmax, j.n);
      kmax = std::max(kmax, j.k);
    }
  const int nj = (int)ord.size();
  SymEigJob *d = dj.ensure(ord.size());
  const void *h = stage ? stage->put(ord.data(), sizeof(SymEigJob) * ord.size()) : ord.data();
  S2G_CUDA(cudaMemcpyAsync(d, h, sizeof(SymEigJob) * ord.size(), cudaMemcpyHostToDevice, s));
  for (int shape = 0, at = 0; shape < kTridiagShapes; at += count[shape++])
    if (count[shape] > 0)
      symeig_tridiag_shape(ord[at].n, [&](int, auto sh) {
        using Shape = decltype(sh);
        launch_cluster(k_symeig_tridiag_b<Shape>, dim3(Shape::C, count[shape]), kTridiagThreads, 0,
                       dim3(Shape::C), s, (const SymEigJob *)(d + at));
      });
  S2G_CUDA(cudaFuncSetAttribute(k_symeig_vectors_b, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)symeig_vec_smem_bytes(kSymEigMaxN)));
  const dim3 g((kmax + kSymEigWarps - 1) / kSymEigWarps, nj);
  S2G_LAUNCH(k_symeig_values_b, dim3(kmax + symeig_bt_blocks(nmax), nj), kValThreads,
             symeig_val_smem_bytes(nmax), s, d);
  S2G_LAUNCH(k_symeig_vectors_b, g, kSymEigWarps * 32, symeig_vec_smem_bytes(nmax), s, d);
  S2G_LAUNCH(k_symeig_backtransform_b, dim3(kmax, nj), kBtThreads, 0, s, d);
}

}  // namespace std2g
