// Blocked Davidson eigensolver for the lowest k roots of the sTDA matrix A.
//
// The reference diagonalises A completely with LAPACK ssyevr and keeps the
// roots in (0, E_thr] (stda.f:1133-1150).  For large CSF spaces this engine
// finds the requested lowest roots iteratively: sigma = A V products through a
// caller-supplied operator (matrix-free, matfree.cuh), and an FP64
// Rayleigh-Ritz projection, FP64 orthogonalisation (classical Gram-Schmidt,
// applied twice) and FP64 residuals.  The preconditioner is the diagonal
// (Davidson) one, (theta - A_ii)^-1.  A few buffer roots beyond the wanted
// ones are carried along so that near-degeneracies at the edge of the wanted
// set do not stall convergence.
#pragma once

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <functional>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "dgemm.cuh"
#include "symeig_seq.cuh"
#include "symeig_small.cuh"

namespace std2g {

// Column norms are reduced in two fixed-order stages so that a block of columns
// spreads over the whole GPU: grid (kColSplit, ncol) writes partial sums of squares,
// which their reader (a kernel, or the host for the residuals) adds in order.
constexpr int kColSplit = 16;

__device__ __forceinline__ double block_sum256(double s, double *red) {
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  return red[0];
}

// R[:, j] -= theta[j] X[:, j]; part[j*gridDim.x + b] = partial |R[:, j]|^2
__global__ void k_dav_resid(double *__restrict__ R, const double *__restrict__ X,
                            const double *__restrict__ theta, int n, double *__restrict__ part) {
  const int j = blockIdx.y;
  const double th = theta[j];
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = chunk * blockIdx.x, i1 = min((int64_t)n, i0 + chunk);
  double s = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    int64_t o = i + (int64_t)n * j;
    double r = R[o] - th * X[o];
    R[o] = r;
    s += r * r;
  }
  __shared__ double red[256];
  s = block_sum256(s, red);
  if (threadIdx.x == 0) part[(int64_t)j * gridDim.x + blockIdx.x] = s;
}

// T[:, j] = R[:, cols[j]] / (theta - diag), guarded away from zero;
// part[j*gridDim.x + b] = partial |T[:, j]|^2 (grid (kColSplit, nc))
__global__ void k_dav_precond(double *__restrict__ T, const double *__restrict__ R,
                              const double *__restrict__ diag, const double *__restrict__ theta,
                              const int *__restrict__ cols, int n, double *__restrict__ part) {
  const int j = blockIdx.y, c = cols[j];
  const double th = theta[c];
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = chunk * blockIdx.x, i1 = min((int64_t)n, i0 + chunk);
  double s = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    double d = th - diag[i];
    if (fabs(d) < 1e-4) d = d < 0 ? -1e-4 : 1e-4;
    const double t = R[i + (int64_t)n * c] / d;
    T[i + (int64_t)n * j] = t;
    s += t * t;
  }
  __shared__ double red[256];
  s = block_sum256(s, red);
  if (threadIdx.x == 0) part[(int64_t)j * gridDim.x + blockIdx.x] = s;
}

// part[j*gridDim.x + b] = partial |T[:, j]|^2
__global__ void k_colnorm_part(const double *__restrict__ T, int n, double *__restrict__ part) {
  const int j = blockIdx.y;
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = chunk * blockIdx.x, i1 = min((int64_t)n, i0 + chunk);
  const double *t = T + (int64_t)n * j;
  double s = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) s += t[i] * t[i];
  __shared__ double red[256];
  s = block_sum256(s, red);
  if (threadIdx.x == 0) part[(int64_t)j * gridDim.x + blockIdx.x] = s;
}

// T[:, j] /= |T[:, j]| from its partial sums of squares (a zero column stays zero);
// grid (any, ncol)
__global__ void k_colnorm_scale(double *__restrict__ T, int n, const double *__restrict__ part,
                                int nsplit) {
  const int j = blockIdx.y;
  double s = 0.0;
  for (int b = 0; b < nsplit; ++b) s += part[(int64_t)j * nsplit + b];
  const double v = sqrt(s), f = v > 0 ? 1.0 / v : 0.0;
  double *t = T + (int64_t)n * j;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    t[i] *= f;
}

// out[j] = sqrt(sum_b part[j*nsplit + b]), in order
__global__ void k_colnorm_finish(const double *__restrict__ part, int nsplit, int ncol,
                                 double *__restrict__ out) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ncol) return;
  double s = 0.0;
  for (int b = 0; b < nsplit; ++b) s += part[(int64_t)j * nsplit + b];
  out[j] = sqrt(s);
}

__global__ void k_unit_vectors(double *__restrict__ V, int n, const int *__restrict__ idx, int k) {
  int64_t total = (int64_t)n * k;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int j = (int)(t / n), i = (int)(t - (int64_t)j * n);
    V[t] = (i == idx[j]) ? 1.0 : 0.0;
  }
}

// T[:, j] *= 1/sqrt(s[j])
__global__ void k_scale_rsqrt(double *__restrict__ T, int n, int ncol,
                              const double *__restrict__ sv) {
  int64_t total = (int64_t)n * ncol;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    double v = sv[t / n];
    T[t] *= v > 0 ? 1.0 / sqrt(v) : 0.0;
  }
}

// H[c + ld*r] = H[r + ld*c] for rows r < m of the new columns c in [m, m+nb)
__global__ void k_mirror_cols(double *__restrict__ H, int ld, int m, int nb) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)m * nb) return;
  int c = m + (int)(t / m), r = (int)(t % m);
  H[c + (int64_t)ld * r] = H[r + (int64_t)ld * c];
}

// H[0:k, 0:k] = diag(theta)
__global__ void k_diag_matrix(double *__restrict__ H, int ld, int k, const double *__restrict__ th) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)k * k) return;
  int c = (int)(t / k), r = (int)(t % k);
  H[r + (int64_t)ld * c] = r == c ? th[r] : 0.0;
}

// Cholesky QR factor of a small Gram matrix, in one CTA: G = L L^T (nc x nc,
// lower triangle read, nc <= kCholMax), then out = L^-T (upper triangular,
// column-major nc x nc, zero below the diagonal) so that T L^-T has
// orthonormal columns.  stat[0] = 1 when a pivot is not positive or its
// square root falls below sqrt(tol) (the block is numerically dependent),
// else 0; stat[1] = the smallest pivot (the diagonal of L).  Deterministic.
// Latency-bound: nc dependent steps.  The elimination runs in place on [G | I]
// in its square-root-free form G = M D M^T: step j subtracts G_ij / d_j times
// row j from every row i > j, over the trailing columns of G and over the
// columns of M^-1 grown so far, which take the places of the eliminated ones.
// Row i lives in the registers of warp i mod 16 (lane = column mod 32); row j
// is passed through shared memory, and the multipliers are its own entries
// (the trailing block is kept whole, hence symmetric), so a step is one read
// of that row, the row updates, one reciprocal (by the lane that holds the next
// pivot) and one barrier.  L^-1 =
// D^-1/2 M^-1 at the end.  10.5 / 21 / 29 / 97 us at nc = 25 / 40 / 62 /
// 112, where a factorisation followed by one forward substitution per thread
// took 29 / 51 / 103 / 333 us.
constexpr int kCholMax = 112;
constexpr int kCholThreads = 512;
template <int RT, int CT>   // rows per warp, columns per lane: nc <= 16 RT, 32 CT
__device__ __forceinline__ void chol_inv_tile(const double *__restrict__ G, int nc, double tol,
                                              double *__restrict__ out, double *__restrict__ stat,
                                              double *row, double *inv, double *piv) {
  constexpr int NW = kCholThreads / 32, LD = 128;   // row: two rows of LD, zero padded
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double w[RT][CT];   // rows i = warp + NW t, columns c = lane + 32 u
#pragma unroll
  for (int t = 0; t < RT; ++t)
#pragma unroll
    for (int u = 0; u < CT; ++u) {
      const int i = warp + NW * t, c = lane + 32 * u;
      w[t][u] = i < nc && c < nc ? G[max(i, c) + nc * min(i, c)] : 0.0;
    }
  for (int q = threadIdx.x; q < 2 * LD; q += kCholThreads) row[q] = 0.0;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int u = 0; u < CT; ++u) row[lane + 32 * u] = w[0][u];
    if (lane == 0) {
      inv[0] = 1.0 / w[0][0];
      piv[0] = w[0][0];
    }
  }
  __syncthreads();
  bool fail = false;
  double dmin = 1e300;
  for (int j = 0; j < nc; ++j) {
    const double *rj = row + (j & 1) * LD;
    const double d = rj[j], di = inv[j & 1];
    double x[CT], m[RT];
#pragma unroll
    for (int u = 0; u < CT; ++u) x[u] = rj[lane + 32 * u];
#pragma unroll
    for (int t = 0; t < RT; ++t) m[t] = warp + NW * t > j ? rj[warp + NW * t] * -di : 0.0;
    // dependent or not positive: the same decision in every thread
    if (!(d > tol) || !(d * d > 0.0) || !isfinite(d)) {
      if (d > 0.0) dmin = fmin(dmin, d);
      fail = true;
      break;
    }
    dmin = fmin(dmin, d);
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
      for (int u = 0; u < CT; ++u) w[t][u] = fma(m[t], x[u], w[t][u]);
    // column j of the rows below becomes M^-1's
#pragma unroll
    for (int u = 0; u < CT; ++u)
      if (lane + 32 * u == j)
#pragma unroll
        for (int t = 0; t < RT; ++t)
          if (warp + NW * t > j) w[t][u] = m[t];
    // the next row, and the reciprocal of its pivot
    if ((j + 1) % NW == warp) {
      double *nx = row + ((j + 1) & 1) * LD;
#pragma unroll
      for (int t = 0; t < RT; ++t)
        if (warp + NW * t == j + 1)
#pragma unroll
          for (int u = 0; u < CT; ++u) {
            nx[lane + 32 * u] = w[t][u];
            if (lane + 32 * u == j + 1) {
              inv[(j + 1) & 1] = 1.0 / w[t][u];
              piv[j + 1] = w[t][u];
            }
          }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    stat[0] = fail ? 1.0 : 0.0;
    stat[1] = dmin < 1e300 ? sqrt(dmin) : dmin;
  }
  if (fail) return;
  // out[c + nc*i] = (L^-1)[i][c]  (upper triangle: c <= i)
#pragma unroll
  for (int t = 0; t < RT; ++t) {
    const int i = warp + NW * t;
    if (i < nc) {
      const double s = 1.0 / sqrt(piv[i]);
#pragma unroll
      for (int u = 0; u < CT; ++u) {
        const int c = lane + 32 * u;
        if (c < nc) out[c + nc * i] = c < i ? w[t][u] * s : (c == i ? s : 0.0);
      }
    }
  }
}

__device__ __forceinline__ void chol_inv_body(const double *__restrict__ G, int nc, double tol,
                                              double *__restrict__ out,
                                              double *__restrict__ stat) {
  __shared__ double row[2 * 128], inv[2], piv[128];
  if (nc <= 32)
    chol_inv_tile<2, 1>(G, nc, tol, out, stat, row, inv, piv);
  else if (nc <= 64)
    chol_inv_tile<4, 2>(G, nc, tol, out, stat, row, inv, piv);
  else
    chol_inv_tile<7, 4>(G, nc, tol, out, stat, row, inv, piv);
}

__global__ void __launch_bounds__(kCholThreads)
k_chol_inv(const double *__restrict__ G, int nc, double tol, double *__restrict__ out,
           double *__restrict__ stat) {
  chol_inv_body(G, nc, tol, out, stat);
}


struct DavidsonWork {
  DBuf<double> V, W, H, Hs, theta, X, R, T, tmp, rn, proj, G, Gc, Gz, lam, work2, part, eigwork,
      stat;
  DBuf<int> cols, idx, info, einfo;   // einfo: of the batched form
  PinnedArena pin;   // small copies from and to the host
  DBuf<double> work;
  int iters = 0;
  int64_t matvecs = 0;
  double max_resid = 0;
  // optional section timing (synchronises at every section boundary):
  // [0] sigma products, [1] projected matrix, [2] its eigen-decomposition,
  // [3] Ritz vectors + residuals, [4] orthogonalisation
  bool profile = false;
  double sec_ms[5] = {0, 0, 0, 0, 0};
  Dgemm *dg = nullptr;   // the context's FP64 products (dgemm.cuh)
  // residual norms and Ritz values of the last Rayleigh-Ritz step (every
  // tracked pair, the buffer roots above the wanted ones included)
  std::vector<double> final_resid, final_theta;
};

// host wall-clock section timer used when DavidsonWork::profile is set
struct SectionClock {
  DavidsonWork &dw;
  cudaStream_t s;
  std::chrono::steady_clock::time_point t0;
  SectionClock(DavidsonWork &w, cudaStream_t st) : dw(w), s(st) {
    if (dw.profile) {
      S2G_CUDA(cudaStreamSynchronize(s));
      t0 = std::chrono::steady_clock::now();
    }
  }
  void tick(int slot) {
    if (!dw.profile) return;
    S2G_CUDA(cudaStreamSynchronize(s));
    auto t1 = std::chrono::steady_clock::now();
    dw.sec_ms[slot] += std::chrono::duration<double, std::milli>(t1 - t0).count();
    t0 = t1;
  }
};

using MatVec = std::function<void(const double *V, int nb, double *W)>;

// Rayleigh-Ritz problems up to this size go to the engine's own eigensolver
// (symeig_small.cuh: 0.10 / 0.22 / 0.66 ms for 16 / 30 / 62 pairs of m = 64 / 120 /
// 300 against 1.1 / 2.3 / 3.2 ms for syevd); larger ones to cuSOLVER syevd.
constexpr int kRRSmallMax = kSymEigMaxN;

// the norm of a column from its kColSplit partial sums of squares
inline double colnorm(const double *part) {
  double s = 0.0;
  for (int b = 0; b < kColSplit; ++b) s += part[b];
  return std::sqrt(s);
}

// order[0..k): the k smallest of n values ascending, ties by index
template <typename Less>
inline std::vector<int> lowest_indices(int n, int k, const Less &less) {
  std::vector<int> order(n);
  std::iota(order.begin(), order.end(), 0);
  std::partial_sort(order.begin(), order.begin() + k, order.end(), [&](int a, int b) {
    return less(a, b) || (!less(b, a) && a < b);
  });
  return order;
}

// Orthonormalises the nc columns of T (n x nc) against the m orthonormal
// columns of V and among themselves, and appends the result to V after column
// m (BCGS2: normalise, then two rounds of one block classical Gram-Schmidt
// projection against V followed by Cholesky QR of the block, or, when its Gram
// matrix is not safely positive definite, orthonormalisation through the Gram
// matrix's eigen-decomposition that drops dependent directions).  dw.part holds
// the partial squared norms of T's columns (kColSplit each).  T may be the place of
// the new columns itself.  Returns the
// number of columns appended, at most `room` (the columns that V can still take):
// a block that is larger goes through the eigen-decomposition, which then keeps its
// leading directions.  kcap: capacity of the k x k work arrays.
// Both rounds of the Cholesky form are issued before the host looks at either's
// status (a failed factor only spoils buffers that the fallback writes anew): one
// wait per block instead of two, each of which left the GPU idle for ~10 us.
// fixed_order: the small factorisations by the kernels of symeig_seq.cuh.
inline int dav_orthonormalize(DavidsonWork &dw, cusolverDnHandle_t sol, cudaStream_t s, double *V, int n, int m, double *T, int nc,
                              int kcap, int room, bool fixed_order = false) {
  const int k = kcap;
  const int grid = 148 * 4;
  const double one = 1.0, zero = 0.0, mone = -1.0;
  if (nc <= 0 || room <= 0) return 0;
  double *tmp = dw.tmp.ensure((size_t)n * k);
  double *proj = dw.proj.ensure((size_t)(m + k) * k + 4);
  double *G = dw.G.ensure((size_t)k * k), *lam = dw.lam.ensure(k);
  double *Li = dw.Gc.ensure((size_t)k * k), *st = dw.stat.ensure(4);
  int *info = dw.info.ensure(1);
  double *dst = V + (size_t)n * m;
  S2G_LAUNCH(k_colnorm_scale, dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(div_up(n, 512), 2 * kColSplit)), (unsigned)nc),
             256, 0, s, T, n, dw.part.get(), kColSplit);
  auto project = [&](double *Tb, int nb) {
    dw.dg->gemm(s, CUBLAS_OP_T, CUBLAS_OP_N, m, nb, n, &one, V, n, Tb, n, &zero, proj, m);
    dw.dg->gemm(s, CUBLAS_OP_N, CUBLAS_OP_N, n, nb, m, &mone, V, n, proj, m, &one, Tb, n);
  };
  auto gram = [&](const double *Tb, int nb) {
    dw.dg->gemm(s, CUBLAS_OP_T, CUBLAS_OP_N, nb, nb, n, &one, Tb, n, Tb, n, &zero, G, nb);
  };
  // Cholesky QR: out = Tb L^-T, its factor from the engine's small factorisation
  auto cholesky = [&](const double *Tb, int nb, double *out, double *stat) {
    if (fixed_order) {
      S2G_CUDA(cudaFuncSetAttribute(seq::k_chol_inv, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(2 * sizeof(double) * kCholMax * kCholMax)));
      S2G_LAUNCH(seq::k_chol_inv, 1, 256, 2 * sizeof(double) * nb * nb, s, G, nb, 1e-8, Li, stat);
    } else {
      S2G_LAUNCH(k_chol_inv, 1, kCholThreads, 0, s, G, nb, 1e-8, Li, stat);
    }
    dw.dg->gemm(s, CUBLAS_OP_N, CUBLAS_OP_N, n, nb, nb, &one, Tb, n, Li, nb, &zero, out, n);
  };
  auto statuses = [&](int count) {   // host copy of st[0 .. 2 count)
    double *h = (double *)dw.pin.take(sizeof(double) * 2 * count);
    S2G_CUDA(cudaMemcpyAsync(h, st, sizeof(double) * 2 * count, cudaMemcpyDeviceToHost, s));
    S2G_CUDA(cudaStreamSynchronize(s));
    dw.pin.reset();
    return h;
  };
  double *Tb = T;
  int ncur = nc, round = 0;
  bool failed = false;   // Tb is projected, and its Gram matrix has no Cholesky factor
  if (nc <= kCholMax && nc <= room && T != dst) {
    for (int r = 0; r < 2; ++r) {
      double *in = r == 0 ? T : tmp, *out = r == 0 ? tmp : dst;
      project(in, nc);
      gram(in, nc);
      cholesky(in, nc, out, st + 2 * r);
    }
    const double *h = statuses(2);
    if (h[0] == 0.0 && h[2] == 0.0) return nc;
    failed = true;
    round = h[0] != 0.0 ? 0 : 1;
    if (round == 1) Tb = tmp;
  }
  for (; round < 2; ++round) {
    if (!failed) project(Tb, ncur);
    gram(Tb, ncur);
    if (!failed && ncur <= kCholMax && ncur <= room) {
      double *o = Tb == dst ? tmp : dst;
      cholesky(Tb, ncur, o, st);
      if (statuses(1)[0] == 0.0) {
        if (o != dst)
          S2G_CUDA(cudaMemcpyAsync(dst, o, sizeof(double) * n * ncur, cudaMemcpyDeviceToDevice, s));
        Tb = dst;
        continue;
      }
    }
    failed = false;
    // eigenpairs of G ascending: drop dependent directions
    if (ncur <= kRRSmallMax) {
      double *Z = dw.Gz.ensure((size_t)k * k);
      S2G_CUDA(cudaMemsetAsync(info, 0, sizeof(int), s));
      if (fixed_order)
        seq::symeig_small(s, G, ncur, ncur, ncur, lam, Z, ncur,
                          dw.eigwork.ensure(seq::symeig_work_doubles(ncur, ncur)), info);
      else
        symeig_small(s, G, ncur, ncur, ncur, lam, Z, ncur,
                     dw.eigwork.ensure(symeig_work_doubles(ncur, ncur)), info);
      S2G_CUDA(cudaMemcpyAsync(G, Z, sizeof(double) * ncur * ncur, cudaMemcpyDeviceToDevice, s));
    } else {
      int lw2 = 0;
      S2G_CUSOLVER(cusolverDnDsyevd_bufferSize(sol, CUSOLVER_EIG_MODE_VECTOR,
                                               CUBLAS_FILL_MODE_LOWER, ncur, G, ncur, lam, &lw2));
      double *work2 = dw.work2.ensure((size_t)lw2 + 1);
      S2G_CUSOLVER(cusolverDnDsyevd(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, ncur,
                                    G, ncur, lam, work2, lw2, info));
    }
    std::vector<double> h_lam(ncur);
    S2G_CUDA(cudaMemcpyAsync(h_lam.data(), lam, sizeof(double) * ncur, cudaMemcpyDeviceToHost, s));
    S2G_CUDA(cudaStreamSynchronize(s));
    int first = 0;   // keep eigenvalues above the dependence threshold
    const double cut = round == 0 ? 1e-10 : 1e-14;
    while (first < ncur && !(h_lam[first] > cut)) ++first;
    first = std::max(first, ncur - room);
    const int nkeep = ncur - first;
    if (nkeep == 0) return 0;
    // new block = Tb U_keep diag(lam_keep)^-1/2, written into V after column m
    double *o = Tb == dst ? tmp : dst;
    dw.dg->gemm(s, CUBLAS_OP_N, CUBLAS_OP_N, n, nkeep, ncur, &one, Tb, n, G + (size_t)ncur * first,
                ncur, &zero, o, n);
    S2G_LAUNCH(k_scale_rsqrt, grid, 256, 0, s, o, n, nkeep, lam + first);
    if (o != dst)
      S2G_CUDA(cudaMemcpyAsync(dst, o, sizeof(double) * n * nkeep, cudaMemcpyDeviceToDevice, s));
    Tb = dst;   // second round re-orthogonalises the appended block in place
    ncur = nkeep;
  }
  return ncur;
}

// Returns the number of converged wanted roots (== k on success).  `mv` forms
// W = A V for nb column vectors (n x nb, column-major); `diag` is diag(A).
// With `warm`, the first block is the k Ritz vectors left in dw.X by a
// previous call on the same problem (orthonormal), instead of unit vectors.
inline int davidson(DavidsonWork &dw, cusolverDnHandle_t sol, cudaStream_t s, const MatVec &mv, const double *diag, int n, int k,
                    double tol, int max_iter, double *omega_out, double *X_out,
                    bool warm = false, bool buffer_roots = true) {
  if (k > n) k = n;
  const int kwant = k;
  // buffer roots (a quarter of the wanted ones, at least 4) and a subspace of
  // up to six blocks, kept within the engine's own Rayleigh-Ritz solver when the
  // block allows: measured against k/2 buffer roots and four blocks, 124 vs
  // 135 ms for the 50 roots of the C384H48 flake, 666 vs 841 ms for 48
  // molecules of 20-150 atoms with 20 roots each
  if (buffer_roots) k = std::min(n, k + std::max(4, k / 4));
  const int mmax = std::min(n, std::max(k + 32, std::min(kSymEigMaxN, 6 * k)));
  const int grid = 148 * 4;
  if (warm && dw.X.n < (size_t)n * k) warm = false;
  double *V = dw.V.ensure((size_t)n * mmax), *W = dw.W.ensure((size_t)n * mmax);
  double *Hs = dw.Hs.ensure((size_t)mmax * mmax);
  double *H = dw.H.ensure((size_t)mmax * mmax);   // V^T W, kept across iterations (ld mmax)
  double *theta = dw.theta.ensure(mmax), *X = dw.X.ensure((size_t)n * k);
  double *R = dw.R.ensure((size_t)n * k), *T = dw.T.ensure((size_t)n * k);
  double *tmp = dw.tmp.ensure((size_t)n * k);
  int *cols = dw.cols.ensure(k);
  // partial squared norms of the residuals, the status of the Rayleigh-Ritz
  // eigensolves behind them: one copy to the host
  double *rpart = dw.rn.ensure((size_t)k * kColSplit + 1);
  int *einfo = (int *)(rpart + (size_t)k * kColSplit);
  dw.part.ensure((size_t)k * kColSplit);
  S2G_CUDA(cudaMemsetAsync(einfo, 0, sizeof(int), s));
  const double one = 1.0, zero = 0.0;

  // initial guess: unit vectors on the k lowest diagonal elements
  std::vector<double> h_diag(n);
  S2G_CUDA(cudaMemcpyAsync(h_diag.data(), diag, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
  S2G_CUDA(cudaStreamSynchronize(s));
  const std::vector<int> order =
      lowest_indices(n, k, [&](int a, int b) { return h_diag[a] < h_diag[b]; });
  int *idx = dw.idx.ensure(k);
  if (warm) {
    S2G_CUDA(cudaMemcpyAsync(V, X, sizeof(double) * n * k, cudaMemcpyDeviceToDevice, s));
  } else {
    S2G_CUDA(cudaMemcpyAsync(idx, order.data(), sizeof(int) * k, cudaMemcpyHostToDevice, s));
    S2G_LAUNCH(k_unit_vectors, grid, 256, 0, s, V, n, idx, k);
  }
  int m = 0, nb = k;
  int lwork = 0;
  if (mmax > kRRSmallMax)
    S2G_CUSOLVER(cusolverDnDsyevd_bufferSize(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                             mmax, Hs, mmax, theta, &lwork));
  double *work = dw.work.ensure((size_t)lwork + 1);
  dw.pin.reset();
  std::vector<double> h_rn(k);
  int nconv = 0;
  dw.iters = 0;
  dw.matvecs = 0;
  SectionClock clk(dw, s);
  for (int it = 0; it < max_iter; ++it) {
    dw.iters = it + 1;
    mv(V + (size_t)n * m, nb, W + (size_t)n * m);
    dw.matvecs += nb;
    clk.tick(0);
    // H = V^T W (ld mmax): only the new columns are formed; the new rows
    // follow from the symmetry of A
    (dw.dg->gemm(s, CUBLAS_OP_T, CUBLAS_OP_N, m + nb, nb, n, &one, V, n,
                           W + (size_t)n * m, n, &zero, H + (size_t)mmax * m, mmax));
    if (m > 0)
      S2G_LAUNCH(k_mirror_cols, (int)div_up((int64_t)m * nb, 256), 256, 0, s, H, mmax, m, nb);
    m += nb;
    clk.tick(1);
    if (m <= kRRSmallMax) {
      // lowest k eigenpairs, eigenvectors into Hs (ld m), no host synchronisation
      symeig_small(s, H, mmax, m, std::min(k, m), theta, Hs, m,
                   dw.eigwork.ensure(symeig_work_doubles(m, std::min(k, m))), einfo);
    } else {
      S2G_CUDA(cudaMemcpy2DAsync(Hs, sizeof(double) * m, H, sizeof(double) * mmax,
                                 sizeof(double) * m, m, cudaMemcpyDeviceToDevice, s));
      S2G_CUSOLVER(cusolverDnDsyevd(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, m, Hs,
                                    m, theta, work, lwork, einfo));
    }
    clk.tick(2);
    // Ritz vectors X = V Y_k, residuals R = W Y_k - X theta: the two products in
    // one launch (members V, W at a fixed distance, which may be negative and leads from
    // one allocation to another: two calls where they go to cuBLAS)
    const auto apart = [](const double *a, const double *b) {
      return (int64_t)((intptr_t)b - (intptr_t)a) / (int64_t)sizeof(double);
    };
    if (dw.dg->lib) {
      dw.dg->run(s, false, false, n, k, m, 1.0, V, n, 0, Hs, m, 0, 0.0, X, n, 0);
      dw.dg->run(s, false, false, n, k, m, 1.0, W, n, 0, Hs, m, 0, 0.0, R, n, 0);
    } else {
      dw.dg->run(s, false, false, n, k, m, 1.0, V, n, apart(V, W), Hs, m, 0, 0.0, X, n, apart(X, R),
                 2);
    }
    S2G_LAUNCH(k_dav_resid, dim3(kColSplit, (unsigned)k), 256, 0, s, R, X, theta, n, rpart);
    const size_t rbytes = sizeof(double) * ((size_t)k * kColSplit + 1);
    const double *h_part = (const double *)dw.pin.take(rbytes);
    S2G_CUDA(cudaMemcpyAsync((void *)h_part, rpart, rbytes, cudaMemcpyDeviceToHost, s));
    S2G_CUDA(cudaStreamSynchronize(s));
    for (int j = 0; j < k; ++j) h_rn[j] = colnorm(h_part + (size_t)j * kColSplit);
    int h_einfo = 0;
    std::memcpy(&h_einfo, h_part + (size_t)k * kColSplit, sizeof(int));
    dw.pin.reset();
    if (h_einfo != 0)
      throw Error{STD2G_ENOCONV, "Davidson: Rayleigh-Ritz eigensolve failed (" +
                                     std::to_string(h_einfo) + ")"};
    std::vector<int> unc;
    int nunc_wanted = 0;
    for (int j = 0; j < k; ++j)
      if (!(h_rn[j] < tol)) {
        unc.push_back(j);
        if (j < kwant) ++nunc_wanted;
      }
    nconv = kwant - nunc_wanted;
    dw.max_resid = *std::max_element(h_rn.begin(), h_rn.begin() + kwant);
    if (dw.profile)
      std::fprintf(stderr, "  davidson iter %d: m %d, unconverged %d of %d, max residual %.3e\n",
                   it + 1, m, nunc_wanted, kwant, dw.max_resid);
    clk.tick(3);
    if (nunc_wanted == 0) break;
    int nc = (int)unc.size();
    S2G_CUDA(cudaMemcpyAsync(cols, dw.pin.put(unc.data(), sizeof(int) * nc), sizeof(int) * nc,
                             cudaMemcpyHostToDevice, s));
    S2G_LAUNCH(k_dav_precond, dim3(kColSplit, (unsigned)nc), 256, 0, s, T, R, diag, theta, cols, n,
               dw.part.get());
    if (m + nc > mmax) {
      // restart with the current Ritz vectors: V <- X, W <- W Y_k
      (dw.dg->gemm(s, CUBLAS_OP_N, CUBLAS_OP_N, n, k, m, &one, W, n, Hs, m, &zero,
                             tmp, n));
      S2G_CUDA(cudaMemcpyAsync(W, tmp, sizeof(double) * n * k, cudaMemcpyDeviceToDevice, s));
      S2G_CUDA(cudaMemcpyAsync(V, X, sizeof(double) * n * k, cudaMemcpyDeviceToDevice, s));
      m = k;
      // H restricted to the Ritz vectors is diag(theta)
      S2G_LAUNCH(k_diag_matrix, (int)div_up((int64_t)k * k, 256), 256, 0, s, H, mmax, k, theta);
    }
    // block orthogonalisation of the corrections, appended to V after column m
    nb = dav_orthonormalize(dw, sol, s, V, n, m, T, nc, k, mmax - m);
    clk.tick(4);
    if (nb == 0) break;
  }
  S2G_CUDA(cudaMemcpyAsync(omega_out, theta, sizeof(double) * kwant, cudaMemcpyDeviceToDevice, s));
  S2G_CUDA(cudaMemcpyAsync(X_out, X, sizeof(double) * n * kwant, cudaMemcpyDeviceToDevice, s));
  dw.final_theta.assign(k, 0.0);
  S2G_CUDA(cudaMemcpyAsync(dw.final_theta.data(), theta, sizeof(double) * k,
                           cudaMemcpyDeviceToHost, s));
  S2G_CUDA(cudaStreamSynchronize(s));
  dw.final_resid = h_rn;
  return nconv;
}

}  // namespace std2g
