// FP64 matrix products of the engine: C = alpha op(A) op(B) + beta C,
// column-major, op = N or T, optionally batched with fixed strides.
//
// B200 has no FP64 kind of tcgen05; its FP64 tensor path is the warp-level
// DMMA (mma.sync m8n8k4 .f64).  Each CTA (4 warps) computes a 64 x BN tile (BN =
// 32 or 64) of C over a K range in steps of 16: the A (64 x 16) and B (16 x BN) tiles
// arrive by 8-byte cp.async in a 4-stage shared-memory ring (three tiles in
// flight while one is multiplied), kept in the global layout's fast order and
// XOR-swizzled so that the fragment reads are conflict-free, and each warp
// owns a 32 x BN/2 sub-tile = 4 x BN/16 DMMA tiles.
//
// Small products and tall-skinny ones (the Davidson projections V^T W: 300 x 75
// outputs over 5e4-long sums) split K across the CTAs of a cluster, which add
// their tiles through distributed shared memory, and across clusters, whose
// partial tiles go to a workspace where the last one to arrive adds them.  Both
// sums run in the order of the splits, so every result is bit-for-bit
// reproducible from run to run.  With beta = 0, C is not read.
#pragma once

#include <cooperative_groups.h>
#include <cublas_v2.h>

#include <algorithm>
#include <vector>

#include "common.cuh"

namespace std2g {

namespace dg {
constexpr int BM = 64, BK = 16, THREADS = 128, STAGES = 4;
constexpr int TILE_A = BM * BK;                              // doubles per A tile
template <int BN> __host__ __device__ constexpr int stage_doubles() { return TILE_A + BN * BK; }
// 64 x 32 tiles: 48 KB (four CTAs per SM); 64 x 64: 64 KB (three)
template <int BN> __host__ __device__ constexpr int smem_bytes() { return STAGES * stage_doubles<BN>() * 8; }
// Shared-memory positions, XOR-swizzled so that the fragment reads of a half
// warp (g = 0..3 along m or n, t = 0..3 along k) hit 16 distinct 8-byte banks:
// operand stored with m (or n) fastest, [BK][W]:
template <int W>
__device__ __forceinline__ int pos_mfast(int k, int m) { return k * W + (m ^ ((k & 3) << 2)); }
// operand stored with k fastest, [rows][BK]:
__device__ __forceinline__ int pos_kfast(int m, int k) { return m * 16 + (k ^ ((m & 3) << 2)); }
}

// D (8x8) += A (8x4, row) * B (4x8, col), FP64.  Fragments: a = A[g][t],
// b = B[t][g], d = {D[g][2t], D[g][2t+1]} with g = lane / 4, t = lane % 4.
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// 8-byte asynchronous global -> shared copy; ok = false fills zeros
__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src),
               "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two-level columns of a product: column n is number n % len of group n / len
// (len = 0: plain columns).  With op(B) = B^T the columns of a group are neighbours: its
// elements of op(B) start at B + n % len + (n / len) sB, and row i of it in C is at
// C + i ldc + n % len + (n / len) sC.  With op(B) = B they are leading dimensions apart:
// B + (n % len) ldb + (n / len) sB and C + i + (n % len) ldc + (n / len) sC.
// The matrix-free products read and write the AOs of one atom in an array over all
// AOs through it.
struct DgSplitCols {
  int len = 0;
  int64_t sB = 0, sC = 0;
  template <bool TB>
  __host__ __device__ __forceinline__ int64_t b(int n, int64_t ldb) const {
    if (len <= 0) return TB ? n : (int64_t)n * ldb;
    return (int64_t)(n % len) * (TB ? 1 : ldb) + (int64_t)(n / len) * sB;
  }
  __host__ __device__ __forceinline__ int64_t c(bool tb, int row, int n, int64_t ldc) const {
    if (len <= 0) return row + (int64_t)n * ldc;
    return (tb ? (int64_t)row * ldc + n % len : row + (int64_t)(n % len) * ldc) +
           (int64_t)(n / len) * sC;
  }
};

// Main loop of one CTA tile: acc = op(A) op(B) over the K range [kb, ke) for
// the 64 x BN tile of C at (m0, n0), shared by the strided-batch kernel
// k_dgemm and the grouped kernel k_dgemm_grouped.
// A tiles are kept in the global layout's fast order: m fastest for op(A) = A
// ([k][m]), k fastest for op(A) = A^T ([m][k]); B tiles k fastest for
// op(B) = B ([n][k]), n fastest for op(B) = B^T ([k][n]); swizzled (pos_*).
// CTA tile 64 x BN (BN = 32, 64); warp w owns rows 32 (w & 1) .. +32 and
// columns (BN / 2)(w >> 1) .. +BN / 2: 4 x BN / 16 DMMA tiles.
template <bool TA, bool TB, int BN>
__device__ __forceinline__ void dgemm_mainloop(int M, int N, const double *__restrict__ A,
                                               int64_t lda, const double *__restrict__ B,
                                               int64_t ldb, int m0, int n0, int kb, int ke,
                                               double *smem_d, double (&acc)[4][BN / 16][2],
                                               const int *__restrict__ bcol = nullptr,
                                               DgSplitCols sc = DgSplitCols{}) {
  using namespace dg;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int NJ = BN / 16, STAGE = stage_doubles<BN>(), TILE_B = BN * BK;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * (BN / 2);
  auto As = [&](int st) { return smem_d + (size_t)st * STAGE; };
  auto Bs = [&](int st) { return smem_d + (size_t)st * STAGE + TILE_A; };

  // Copies of one K tile into a stage: element q of this thread is tid + 128 q,
  // each with its own source pointer that moves on by one K tile per call.  Rows
  // past M (columns past N) read the last valid one instead: they only reach
  // outputs that are not stored, so a full K tile needs no test at all; the
  // last, partial K tile is filled with zeros past ke.  With one CTA on an SM
  // a K tile costs what its instructions take to issue (272 of them per warp
  // with tests and addresses formed per copy took 1040 cycles, twice the 512
  // of the DMMAs).
  constexpr int QA = TILE_A / THREADS, QB = TILE_B / THREADS, KS = THREADS / BN;
  const double *pa[QA], *pb[QB];
  const int ka = TA ? tid & 15 : tid >> 6, kbq = TB ? tid / BN : tid & 15;
#pragma unroll
  for (int q = 0; q < QA; ++q)
    pa[q] = TA ? A + (kb + ka) + (int64_t)min(m0 + (tid >> 4) + 8 * q, M - 1) * lda
               : A + min(m0 + (tid & 63), M - 1) + (int64_t)(kb + ka + 2 * q) * lda;
#pragma unroll
  for (int q = 0; q < QB; ++q) {
    if (TB) {
      pb[q] = B + sc.b<true>(min(n0 + (tid & (BN - 1)), N - 1), ldb) + (int64_t)(kb + kbq + KS * q) * ldb;
    } else {   // bcol: column n of op(B) is column bcol[n] of B
      const int n = min(n0 + (tid >> 4) + 8 * q, N - 1);
      pb[q] = B + (kb + kbq) + sc.b<false>(bcol ? bcol[n] : n, ldb);
    }
  }
  const int64_t sa = TA ? BK : BK * lda, sb = TB ? BK * ldb : BK;
  auto issue = [&](int st, int left) {   // left: K elements from the tile's start to ke
    double *a = As(st), *b = Bs(st);
    auto dst_a = [&](int q) {
      return TA ? a + pos_kfast((tid >> 4) + 8 * q, ka) : a + pos_mfast<BM>(ka + 2 * q, tid & 63);
    };
    auto dst_b = [&](int q) {
      return TB ? b + pos_mfast<BN>(kbq + KS * q, tid & (BN - 1))
                : b + pos_kfast((tid >> 4) + 8 * q, kbq);
    };
    if (left >= BK) {
#pragma unroll
      for (int q = 0; q < QA; ++q) cp_async8(dst_a(q), pa[q]);
#pragma unroll
      for (int q = 0; q < QB; ++q) cp_async8(dst_b(q), pb[q]);
    } else {
#pragma unroll
      for (int q = 0; q < QA; ++q) {
        const bool ok = ka + (TA ? 0 : 2 * q) < left;
        cp_async8(dst_a(q), ok ? pa[q] : A, ok);
      }
#pragma unroll
      for (int q = 0; q < QB; ++q) {
        const bool ok = kbq + (TB ? KS * q : 0) < left;
        cp_async8(dst_b(q), ok ? pb[q] : B, ok);
      }
    }
#pragma unroll
    for (int q = 0; q < QA; ++q) pa[q] += sa;
#pragma unroll
    for (int q = 0; q < QB; ++q) pb[q] += sb;
  };

#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int nt = ke > kb ? (ke - kb + BK - 1) / BK : 0;
#pragma unroll
  for (int p = 0; p < STAGES - 1; ++p) {
    if (p < nt) issue(p, ke - kb - p * BK);
    cp_async_commit();
  }
  for (int it = 0; it < nt; ++it) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    {
      const int nx = it + STAGES - 1;
      if (nx < nt) issue(nx % STAGES, ke - kb - nx * BK);
      cp_async_commit();
    }
    const double *a = As(it % STAGES), *b = Bs(it % STAGES);
#pragma unroll
    for (int ks = 0; ks < BK; ks += 4) {
      double fa[4], fb[NJ];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = wm + 8 * i + g, k = ks + t;
        fa[i] = TA ? a[pos_kfast(m, k)] : a[pos_mfast<BM>(k, m)];
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int n = wn + 8 * j + g, k = ks + t;
        fb[j] = TB ? b[pos_mfast<BN>(k, n)] : b[pos_kfast(n, k)];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], fa[i], fb[j]);
    }
  }
  cp_async_wait<0>();
}

// blockIdx.x: tile of C (m fastest, or n fastest); blockIdx.y: batch * ksplit + split.
// Each split covers K range [split * kchunk, min(K, (split + 1) * kchunk)).
// ksplit == 1: C = alpha acc + beta C.
// arrived == NULL: work[(b * ksplit + split)][m + n M] = acc (k_dgemm_reduce).
// Otherwise the cs consecutive splits of a cluster (cluster 1 x cs) are added
// through distributed shared memory, CTA r taking slice r of the tile's
// elements; with more than one cluster per tile each writes its sum to
// work[tile][cluster][element], and the CTA that arrives last at the slice's
// counter adds them in order, stores C and resets the counter.
template <bool TA, bool TB, int BN>
__global__ void __launch_bounds__(dg::THREADS, BN == 32 ? 4 : 3)
    k_dgemm(int M, int N, int K, double alpha, const double *__restrict__ A, int64_t lda,
            int64_t sA, const double *__restrict__ B, int64_t ldb, int64_t sB, double beta,
            double *__restrict__ C, int64_t ldc, int64_t sC, int ksplit, int kchunk,
            double *__restrict__ work, int tri, int nfast, int cs, int *__restrict__ arrived,
            DgSplitCols sc) {
  using namespace dg;
  extern __shared__ __align__(16) double smem_d[];
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int m0 = (nfast ? blockIdx.x / tiles_n : blockIdx.x % tiles_m) * BM;
  const int n0 = (nfast ? blockIdx.x % tiles_n : blockIdx.x / tiles_m) * BN;
  // tri > 0: column n is the pair (i, j) = (n / tri, n % tri) of a symmetric
  // pair array and only j <= i is wanted: a tile whose columns all lie above
  // the diagonal is skipped (the caller mirrors those columns)
  if (tri > 0) {
    const int i0 = n0 / tri, i1 = min(N - 1, n0 + BN - 1) / tri;
    if (i0 == i1 && n0 - i0 * tri > i0) return;   // the same in the whole cluster
  }
  // tri < 0: the product is symmetric; tiles above the diagonal are skipped and
  // the elements below it written to both places
  if (tri < 0 && n0 >= m0 + BM) return;
  const int batch = blockIdx.y / ksplit, split = blockIdx.y % ksplit;
  const int kb = split * kchunk, ke = min(K, kb + kchunk);
  A += batch * sA;
  B += batch * sB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int NJ = BN / 16;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * (BN / 2);
  double acc[4][NJ][2];
  dgemm_mainloop<TA, TB, BN>(M, N, A, lda, B, ldb, m0, n0, kb, ke, smem_d, acc, nullptr, sc);

  // epilogue: element (i, j, e) of this thread is C[m0 + wm + 8 i + g][n0 + wn + 8 j + 2 t + e]
  C += batch * sC;
  auto store = [&](int row, int col, double s) {
    if (tri < 0 && row < col) return;
    double *p = C + sc.c(TB, row, col, ldc);
    const double v = alpha * s, x = beta == 0.0 ? v : v + beta * *p;
    *p = x;
    if (tri < 0) C[col + (int64_t)row * ldc] = x;
  };
  if (ksplit == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = m0 + wm + 8 * i + g;
      if (row >= M) continue;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = n0 + wn + 8 * j + 2 * t + e;
          if (col < N) store(row, col, acc[i][j][e]);
        }
    }
  } else if (!arrived) {
    double *wp = work + (int64_t)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = m0 + wm + 8 * i + g;
      if (row >= M) continue;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = n0 + wn + 8 * j + 2 * t + e;
          if (col < N) wp[row + (int64_t)col * M] = acc[i][j][e];
        }
    }
  } else {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int LD = BM + 4;   // the tile in shared memory, column-major
    static_assert(LD * BN <= STAGES * stage_doubles<BN>(), "tile in the pipeline's memory");
    __syncthreads();             // the last stage has been read
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          smem_d[(wn + 8 * j + 2 * t + e) * LD + wm + 8 * i + g] = acc[i][j][e];
    cl.sync();
    constexpr int E = BM * BN;
    const int rank = split % cs, ng = ksplit / cs, per = E / cs, tiles = gridDim.x;
    const int64_t tile = (int64_t)batch * tiles + blockIdx.x;
    double *wp = work + tile * ng * E;   // [cluster][element]
    const double *remote[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) remote[r] = r < cs ? cl.map_shared_rank(smem_d, r) : smem_d;
#pragma unroll 4
    for (int x = tid; x < per; x += THREADS) {
      const int el = rank * per + x, at = (el / BM) * LD + el % BM;
      double v[8], s = 0.0;
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = r < cs ? remote[r][at] : 0.0;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < cs) s += v[r];
      if (ng == 1) {
        const int row = m0 + el % BM, col = n0 + el / BM;
        if (row < M && col < N) store(row, col, s);
      } else {
        wp[(int64_t)(split / cs) * E + el] = s;
      }
    }
    cl.sync();   // no CTA leaves while others may still read its tile
    if (ng > 1) {
      __shared__ int last;
      __threadfence();
      __syncthreads();
      if (tid == 0) last = atomicAdd(arrived + tile * cs + rank, 1) == ng - 1;
      __syncthreads();
      if (last) {
        __threadfence();
        for (int x = tid; x < per; x += THREADS) {
          const int el = rank * per + x, row = m0 + el % BM, col = n0 + el / BM;
          double s = 0.0;
          for (int q = 0; q < ng; q += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = q + u < ng ? __ldcg(wp + (int64_t)(q + u) * E + el) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (q + u < ng) s += v[u];
          }
          if (row < M && col < N) store(row, col, s);
        }
        if (tid == 0) arrived[tile * cs + rank] = 0;
      }
    }
  }
}

// s + w[0] + w[mn] + ... + w[(ks-1) mn], added in that order; the loads go out 16
// at a time, so that the sum costs a few memory latencies instead of ks / 4
__device__ __forceinline__ double split_sum(const double *__restrict__ w, int64_t mn, int ks) {
  double s = 0.0;
  int q = 0;
  for (; q + 16 <= ks; q += 16) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = w[(q + u) * mn];
#pragma unroll
    for (int u = 0; u < 16; ++u) s += v[u];
  }
  double v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) v[u] = q + u < ks ? w[(q + u) * mn] : 0.0;
#pragma unroll
  for (int u = 0; u < 16; ++u)
    if (q + u < ks) s += v[u];
  return s;
}

// C = alpha sum_s work[b][s] + beta C, splits added in order 0, 1, ...
constexpr int kReduceThreads = 64;   // few outputs: small blocks reach more SMs
__global__ void __launch_bounds__(kReduceThreads)
k_dgemm_reduce(int M, int N, int batch, int ksplit, double alpha, const double *__restrict__ work,
               double beta, double *__restrict__ C, int64_t ldc, int64_t sC, DgSplitCols sc,
               bool tb) {
  const int64_t mn = (int64_t)M * N, total = mn * batch;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total;
       x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = x / mn, r = x - b * mn;
    const int64_t col = r / M, row = r - col * M;
    const double s = split_sum(work + b * ksplit * mn + r, mn, ksplit);
    double *p = C + b * sC + sc.c(tb, (int)row, (int)col, ldc);
    *p = beta == 0.0 ? alpha * s : alpha * s + beta * *p;
  }
}

// For products on cuBLAS: P[k + K (n + N q)] = element (k, n) of member q's op(B) with
// two-level columns, or with column n at cols[n], and back: C = P + beta C on its columns
__global__ void k_dgemm_pack(double *__restrict__ P, const double *__restrict__ B, int64_t ldb,
                             int64_t sB, int N, int K, int batch, bool tb, DgSplitCols sc,
                             const int *__restrict__ cols) {
  const int64_t total = (int64_t)K * N * batch;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total;
       x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = x / K, q = c / N;
    const int k = (int)(x - c * K), at = (int)(c - q * N), n = cols ? cols[at] : at;
    P[x] = B[q * sB + (tb ? sc.b<true>(n, ldb) + k * ldb : sc.b<false>(n, ldb) + k)];
  }
}
__global__ void k_dgemm_spread(double *__restrict__ C, int64_t ldc, int64_t sC,
                               const double *__restrict__ P, int M, int N, int batch, bool tb,
                               DgSplitCols sc, const int *__restrict__ cols, double beta) {
  const int64_t total = (int64_t)M * N * batch;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total;
       x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = x / M, q = c / N;
    const int i = (int)(x - c * M), at = (int)(c - q * N), n = cols ? cols[at] : at;
    double *p = C + q * sC + sc.c(tb, i, n, ldc);
    *p = beta == 0.0 ? P[x] : P[x] + beta * *p;
  }
}

// One member of a grouped launch: C = alpha op(A) op(B) + beta C with op(A)
// M x K and op(B) K x N (column-major; beta = 0: C is not read).
struct DgProblem {
  int M, N, K;
  double alpha, beta;
  const double *A, *B;
  double *C;
  int64_t lda, ldb, ldc;
  // columns by index (op(B) = B only): column n of op(B) is column bcol[n] of B,
  // column n of C is column ccol[n] of the array at C
  const int *bcol = nullptr, *ccol = nullptr;
  int ks = 1;          // K splits (set by Dgemm::grouped)
  int64_t woff = 0;    // the member's partial tiles in the workspace (ks > 1)
};

// Products of different shapes and operands in one launch (one op(A), op(B)
// and tile width for all): blockIdx.x runs over the tiles of every member,
// member p owning tiles [tile0[p], tile0[p + 1]) (m fastest, then the K
// split); a binary search maps the CTA to its member.  A member with ks > 1
// splits K into ks ranges whose partial tiles go to work + woff and are added
// in split order by k_dgemm_grouped_reduce (deterministic, no atomics).
template <bool TA, bool TB, int BN>
__global__ void __launch_bounds__(dg::THREADS, BN == 32 ? 4 : 3)
    k_dgemm_grouped(const DgProblem *__restrict__ probs, const int *__restrict__ tile0,
                    int nprob, double *__restrict__ work) {
  using namespace dg;
  extern __shared__ __align__(16) double smem_d[];
  const int tb = blockIdx.x;
  int lo = 0, hi = nprob;   // tile0[lo] <= tb < tile0[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile0[mid] <= tb) lo = mid;
    else hi = mid;
  }
  const DgProblem pr = probs[lo];
  const int tiles_m = (pr.M + BM - 1) / BM, tiles_mn = tiles_m * ((pr.N + BN - 1) / BN);
  const int local = (tb - tile0[lo]) % tiles_mn, split = (tb - tile0[lo]) / tiles_mn;
  const int m0 = (local % tiles_m) * BM, n0 = (local / tiles_m) * BN;
  const int kchunk = (((pr.K + pr.ks - 1) / pr.ks + BK - 1) / BK) * BK;
  const int kb = split * kchunk, ke = min(pr.K, kb + kchunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  constexpr int NJ = BN / 16;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * (BN / 2);
  double acc[4][NJ][2];
  dgemm_mainloop<TA, TB, BN>(pr.M, pr.N, pr.A, pr.lda, pr.B, pr.ldb, m0, n0, kb, ke, smem_d,
                             acc, pr.bcol);
  double *wp = work + pr.woff + (int64_t)split * pr.M * pr.N;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + wm + 8 * i + g;
    if (row >= pr.M) continue;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = n0 + wn + 8 * j + 2 * t + e;
        if (col >= pr.N) continue;
        if (pr.ks > 1) {
          wp[row + (int64_t)col * pr.M] = acc[i][j][e];
        } else {
          double *p = pr.C + row + (int64_t)(pr.ccol ? pr.ccol[col] : col) * pr.ldc;
          const double v = pr.alpha * acc[i][j][e];
          *p = pr.beta == 0.0 ? v : v + pr.beta * *p;
        }
      }
  }
}

// C = alpha sum_s work[woff + s M N] + beta C for the members with ks > 1
// (blockIdx.y = member), splits added in order 0, 1, ...
__global__ void k_dgemm_grouped_reduce(const DgProblem *__restrict__ probs,
                                       const double *__restrict__ work) {
  const DgProblem pr = probs[blockIdx.y];
  if (pr.ks <= 1) return;
  const int64_t mn = (int64_t)pr.M * pr.N;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < mn;
       x += (int64_t)gridDim.x * blockDim.x) {
    const double s = split_sum(work + pr.woff + x, mn, pr.ks);
    const int64_t col = x / pr.M, row = x - col * pr.M;
    double *p = pr.C + row + col * pr.ldc;
    *p = pr.beta == 0.0 ? pr.alpha * s : pr.alpha * s + pr.beta * *p;
  }
}

// Launch wrapper with the split-K workspace.
struct Dgemm {
  DBuf<double> work;
  DBuf<int> arrived;   // arrival counters of the split tiles (one stream per instance)
  int nsm = 148;
  int64_t launches = 0;
  // set: the products go to cuBLAS on this handle instead (the library
  // baseline of the plain FP64 form, STD2G_FLAG_LIBRARY_FP64)
  cublasHandle_t lib = nullptr;
  DBuf<double> packed;   // two-level columns and results of those products, contiguous
  // per-product device time (an event pair around each product) and the
  // algorithmic FLOPs 2 m n k of the products since the last reset()
  bool timed = false;
  std::vector<cudaEvent_t> ev;
  size_t nev = 0;
  double flop = 0;
  int64_t calls = 0;
  ~Dgemm() {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
  }
  void reset() {
    nev = 0;
    flop = 0;
    calls = 0;
    launches = 0;
  }
  // event pair around one product or grouped launch, where they are timed
  struct Timed {
    Dgemm &g;
    cudaStream_t s;
    Timed(Dgemm &dg, cudaStream_t stream) : g(dg), s(stream) {
      if (g.timed) g.mark(s);
    }
    ~Timed() {
      try {
        if (g.timed) g.mark(s);
      } catch (const Error &) {   // the launch's own error is the one to report
      }
    }
  };
  // device time of the timed products since reset(); the stream must have
  // passed them (the caller synchronises first)
  double elapsed_ms() const {
    double ms = 0;
    for (size_t q = 0; q + 1 < nev; q += 2) {
      float t = 0;
      if (cudaEventElapsedTime(&t, ev[q], ev[q + 1]) == cudaSuccess) ms += t;
    }
    return ms;
  }
  void mark(cudaStream_t s) {
    if (nev == ev.size()) {
      cudaEvent_t e;
      S2G_CUDA(cudaEventCreate(&e));
      ev.push_back(e);
    }
    S2G_CUDA(cudaEventRecord(ev[nev++], s));
  }

  // grouped launch (k_dgemm_grouped) of the members with a non-empty output, in
  // tiles of 64 columns where those fill the GPU, else of 32; the descriptors
  // go to `gdesc` / `gtile0` (same stream: a later launch's upload waits for this
  // launch), from `stage` when given
  DBuf<DgProblem> gdesc;
  DBuf<int> gtile0;
  DBuf<double> gwork;   // partial tiles of the split members
  void grouped(cudaStream_t s, bool ta, bool tb, const std::vector<DgProblem> &in,
               PinnedArena *stage = nullptr) {
    if (lib) return library_grouped(s, ta, tb, in);
    std::vector<DgProblem> pr;
    std::vector<int> t0(1, 0);
    int64_t wtot = 0;
    int64_t mnmax = 0;
    int64_t t64 = 0;
    bool split = false;
    for (const DgProblem &q : in) {
      if (q.M <= 0 || q.N <= 0) continue;
      t64 += div_up(q.M, dg::BM) * div_up(q.N, 64);
      split |= !q.ccol && q.K >= 512;
    }
    const int bn = !split && t64 >= 3 * (int64_t)nsm ? 64 : 32;
    for (DgProblem q : in) {
      if (q.M <= 0 || q.N <= 0) continue;
      // long sums over few output tiles (the Davidson's projections, A V of
      // a small block) split K: at least 256 per split, about 128 CTAs
      const int64_t tmn = div_up(q.M, dg::BM) * div_up(q.N, bn);
      q.ks = q.ccol ? 1
                    : (int)std::max<int64_t>(1, std::min<int64_t>({32, q.K / 256,
                                                                   std::max<int64_t>(1, 128 / tmn)}));
      q.woff = wtot;
      if (q.ks > 1) wtot += (int64_t)q.ks * q.M * q.N;
      mnmax = std::max<int64_t>(mnmax, (int64_t)q.M * q.N);
      pr.push_back(q);
      t0.push_back(t0.back() + (int)(tmn * q.ks));
      flop += 2.0 * q.M * q.N * (double)q.K;
    }
    if (pr.empty()) return;
    ++calls;
    Timed around(*this, s);
    const int np = (int)pr.size();
    double *wk = wtot > 0 ? gwork.ensure((size_t)wtot) : nullptr;
    DgProblem *d = gdesc.ensure(pr.size());
    int *dt = gtile0.ensure(t0.size());
    const void *hp = pr.data(), *ht = t0.data();
    if (stage) {
      hp = stage->put(pr.data(), sizeof(DgProblem) * pr.size());
      ht = stage->put(t0.data(), sizeof(int) * t0.size());
    }
    S2G_CUDA(cudaMemcpyAsync(d, hp, sizeof(DgProblem) * pr.size(), cudaMemcpyHostToDevice, s));
    S2G_CUDA(cudaMemcpyAsync(dt, ht, sizeof(int) * t0.size(), cudaMemcpyHostToDevice, s));
#define S2G_DGEMM_G(TA_, TB_, BN_)                                                              \
  do {                                                                                          \
    S2G_CUDA(cudaFuncSetAttribute(k_dgemm_grouped<TA_, TB_, BN_>,                               \
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,                  \
                                  dg::smem_bytes<BN_>()));                                      \
    S2G_LAUNCH((k_dgemm_grouped<TA_, TB_, BN_>), t0.back(), dg::THREADS, dg::smem_bytes<BN_>(), \
               s, d, dt, np, wk);                                                               \
  } while (0)
    if (bn == 64) {
      if (!ta && !tb) S2G_DGEMM_G(false, false, 64);
      else if (ta && !tb) S2G_DGEMM_G(true, false, 64);
      else if (!ta && tb) S2G_DGEMM_G(false, true, 64);
      else S2G_DGEMM_G(true, true, 64);
    } else {
      if (!ta && !tb) S2G_DGEMM_G(false, false, 32);
      else if (ta && !tb) S2G_DGEMM_G(true, false, 32);
      else if (!ta && tb) S2G_DGEMM_G(false, true, 32);
      else S2G_DGEMM_G(true, true, 32);
    }
#undef S2G_DGEMM_G
    ++launches;
    if (wtot > 0) {
      const int g = (int)std::max<int64_t>(1, std::min<int64_t>(div_up(mnmax, 256), 64));
      S2G_LAUNCH(k_dgemm_grouped_reduce, dim3(g, np), 256, 0, s, d, wk);
      ++launches;
    }
  }

  // this instance's launches have set the kernels' shared-memory limits (a
  // host call per product otherwise; an instance serves one device)
  bool smem_set[2][2][2] = {};
  // K splits by wave counts only (see pick_split): the sTD-DFT subspace
  // iteration, whose results must not depend on the order of these sums
  bool wave_splits = false;

  // Tile width, cluster size and clusters per tile of one product, by the time
  // (us) of the busiest SM: every product starts and stores in ~3.9; a K step of
  // 16 is bound by the DMMA rate (64 FMA per SM and cycle) and takes 0.31 / 0.54
  // for BN = 32 / 64, counted over the CTAs that share the busiest SM and not over
  // those that fit on it (300 CTAs on 148 SMs take half as long again as 296).  A
  // CTA alone on its SM has one warp per scheduler, which issues a DMMA only every
  // ~30 cycles instead of 16, so it counts for two.  Adding the tiles of a cluster
  // takes 1.6 + 5.5 / cs, adding g clusters 1 + 0.23 g more (per 32 columns);
  // several clusters are full ones, so that eight CTAs share the last sum, and
  // about 0.86 of the slots can hold clusters at a time.  Fitted to sweeps of 66
  // products of the solver, where it picks a shape within 15 % of the best one in
  // all but three: 220^3 13.5 -> 8.4 us with 8 CTAs per tile, 75 x 25 x 5945
  // (transposed) 16.6 -> 12.7 us, against one CTA per tile or split sums in a
  // second launch.  (Tiles of 128 columns were 3 to 8 % slower than 64 wherever
  // they fill the GPU: 432 x 100000 x 432 1265 against 1181 us.)
  // wave_splits: the split count by waves of four 64 x 32, three 64 x 64 or two
  // 64 x 128 CTAs per SM, the fewest K steps of the busiest SM (splits at least
  // 256 long, weighted 3 %), a step of a full wave taking 0.74 / 1 / 1.31; no
  // clusters.  The tile's width does not change a sum.
  void pick_split(int m, int n, int k, int batch, bool sym, int &bn, int &ksplit,
                  int &cs) const {
    double best = 0.0;
    const int64_t kk = std::max(k, 1), tm = div_up(m, dg::BM);
    auto tiles_of = [&](int w) {
      return (sym ? tm * (tm + 1) / 2 * (dg::BM / w) : tm * div_up(n, w)) * (int64_t)batch;
    };
    if (wave_splits) {
      const int kmax = (int)std::max<int64_t>(1, std::min<int64_t>(64, k / 256));
      for (int w : {32, 64, 128}) {
        const int64_t slots = (w == 32 ? 4 : (w == 64 ? 3 : 2)) * (int64_t)nsm;
        const double wave_step = w == 32 ? 0.74 : (w == 64 ? 1.0 : 1.31);
        for (int ks = 1; ks <= kmax; ++ks) {
          const int64_t steps =
              div_up(tiles_of(w) * ks, slots) * div_up(div_up(kk, ks), dg::BK);
          const double cost = (double)steps * wave_step * (ks > 1 ? 1.03 : 1.0);
          if (best == 0.0 || cost < best) {
            best = cost;
            bn = std::min(w, 64);
            ksplit = ks;
          }
        }
      }
      cs = 0;
      return;
    }
    for (int w : {32, 64}) {
      const int64_t ctas = tiles_of(w), resident = w == 32 ? 4 : 3, slots = resident * nsm;
      const double step = w == 32 ? 0.31 : 0.54, cols = w / 32.0;
      for (int c : {1, 2, 4, 8})
        for (int g : {1, 2, 3, 4, 6, 8, 12, 16, 24}) {
          const int64_t ks = (int64_t)c * g;
          // no split shorter than a K step, or of a product that fills the GPU
          if ((g > 1 && c < 8) || (ks > 1 && ((ks - 1) * dg::BK >= kk || ctas >= slots))) break;
          const int64_t kt = div_up(div_up(kk, ks), dg::BK);
          const int64_t room = c > 1 ? slots * 86 / 100 : slots;
          const int64_t full = (ctas * ks - 1) / room, q = div_up(ctas * ks - full * room, nsm);
          const double cost =
              (double)kt * step * (double)(full * resident) +
              (double)kt * step * (q == 1 ? 2.05 : (double)q) + (c > 1 ? 12.0 : 0.8) * (double)full +
              (c > 1 ? 1.6 + 5.5 * cols / c : 0.0) + (g > 1 ? 1.0 + 0.23 * g * cols : 0.0);
          if (best == 0.0 || cost < best) {
            best = cost;
            bn = w;
            ksplit = (int)ks;
            cs = c;
          }
        }
    }
  }

  // the argument order of cublasDgemm (alpha / beta by pointer, host values)
  void gemm(cudaStream_t s, cublasOperation_t ta, cublasOperation_t tb, int m, int n, int k,
            const double *alpha, const double *A, int64_t lda, const double *B, int64_t ldb,
            const double *beta, double *C, int64_t ldc) {
    run(s, ta != CUBLAS_OP_N, tb != CUBLAS_OP_N, m, n, k, *alpha, A, lda, 0, B, ldb, 0, *beta, C,
        ldc, 0, 1);
  }

  // run() on cuBLAS: the whole product where `tri` asks for a part of it (the rest
  // is what the caller would mirror).  Two-level columns are packed into one block per
  // member before, and the result is spread after it, outside the timed region (one
  // strided batch per group of 4 columns halved the rate over C384H48's products).
  void library(cudaStream_t s, bool ta, bool tb, int m, int n, int k, double alpha,
               const double *A, int64_t lda, int64_t sA, const double *B, int64_t ldb, int64_t sB,
               double beta, double *C, int64_t ldc, int64_t sC, int batch, DgSplitCols sc) {
    S2G_CUBLAS(cublasSetStream(lib, s));
    auto product = [&](cublasOperation_t ob, const double *Y, int64_t ldy, int64_t sY, double bt,
                       double *Z, int64_t ldz, int64_t sZ) {
      Timed around(*this, s);
      const cublasOperation_t oa = ta ? CUBLAS_OP_T : CUBLAS_OP_N;
      if (batch == 1)
        S2G_CUBLAS(cublasDgemm(lib, oa, ob, m, n, k, &alpha, A, (int)lda, Y, (int)ldy, &bt, Z,
                               (int)ldz));
      else
        S2G_CUBLAS(cublasDgemmStridedBatched(lib, oa, ob, m, n, k, &alpha, A, (int)lda, sA, Y,
                                             (int)ldy, sY, &bt, Z, (int)ldz, sZ, batch));
    };
    if (sc.len <= 0) {
      product(tb ? CUBLAS_OP_T : CUBLAS_OP_N, B, ldb, sB, beta, C, ldc, sC);
      return;
    }
    const int64_t kn = (int64_t)k * n, mn = (int64_t)m * n;
    double *Bp = packed.ensure((size_t)batch * (kn + mn)), *Cp = Bp + batch * kn;
    const int g = nsm * 16;
    S2G_LAUNCH(k_dgemm_pack, g, 256, 0, s, Bp, B, ldb, sB, n, k, batch, tb, sc, nullptr);
    product(CUBLAS_OP_N, Bp, k, kn, 0.0, Cp, m, mn);
    S2G_LAUNCH(k_dgemm_spread, g, 256, 0, s, C, ldc, sC, Cp, m, n, batch, tb, sc, nullptr, beta);
  }

  // grouped() on cuBLAS: one call per member, indexed columns packed and spread
  void library_grouped(cudaStream_t s, bool ta, bool tb, const std::vector<DgProblem> &in) {
    const int g = nsm * 16;
    for (const DgProblem &q : in) {
      if (q.M <= 0 || q.N <= 0) continue;
      flop += 2.0 * q.M * q.N * (double)q.K;
      ++calls;
      const int64_t kn = (int64_t)q.K * q.N, mn = (int64_t)q.M * q.N;
      double *Bp = q.bcol || q.ccol ? packed.ensure((size_t)(kn + mn)) : nullptr, *Cp = Bp + kn;
      const double *B = q.B;
      int64_t ldb = q.ldb;
      if (q.bcol) {   // op(B) = B
        S2G_LAUNCH(k_dgemm_pack, g, 256, 0, s, Bp, q.B, q.ldb, (int64_t)0, q.N, q.K, 1, false,
                   DgSplitCols{}, q.bcol);
        B = Bp;
        ldb = q.K;
      }
      library(s, ta, tb, q.M, q.N, q.K, q.alpha, q.A, q.lda, 0, B, ldb, 0, q.ccol ? 0.0 : q.beta,
              q.ccol ? Cp : q.C, q.ccol ? q.M : q.ldc, 0, 1, DgSplitCols{});
      if (q.ccol)
        S2G_LAUNCH(k_dgemm_spread, g, 256, 0, s, q.C, q.ldc, (int64_t)0, Cp, q.M, q.N, 1, false,
                   DgSplitCols{}, q.ccol, q.beta);
    }
  }

  // op(A) is m x k, op(B) is k x n; strides between batch members (0 for one).
  // tri > 0: see k_dgemm; tri < 0: a symmetric n x n result (not with wave_splits).
  // sc: two-level columns.
  void run(cudaStream_t s, bool ta, bool tb, int m, int n, int k, double alpha, const double *A,
           int64_t lda, int64_t sA, const double *B, int64_t ldb, int64_t sB, double beta,
           double *C, int64_t ldc, int64_t sC, int batch = 1, int tri = 0,
           DgSplitCols sc = DgSplitCols{}) {
    if (sc.len > 0 && tri != 0) throw Error{STD2G_EINVAL, "dgemm: split columns"};
    // (its split sums in a second launch would take in tiles that are not formed)
    if (tri < 0 && wave_splits) throw Error{STD2G_EINVAL, "dgemm: symmetric result"};
    if (m <= 0 || n <= 0 || batch <= 0) return;
    if (k < 0) throw Error{STD2G_EINVAL, "dgemm: negative k"};
    flop += 2.0 * m * n * (double)k * batch;
    ++calls;
    if (lib) {
      library(s, ta, tb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, sc);
      return;
    }
    Timed around(*this, s);
    int bn = 64, ksplit = 1, cs = 1;
    pick_split(m, n, k, batch, tri < 0, bn, ksplit, cs);
    const int tiles = (int)(div_up(m, dg::BM) * div_up(n, bn));
    const int kchunk = (int)div_up(div_up(std::max(k, 1), ksplit), dg::BK) * dg::BK;
    if (cs == 0) ksplit = (int)div_up(std::max(k, 1), kchunk);
    if (batch * ksplit > 65535) throw Error{STD2G_EINVAL, "dgemm: batch too large"};
    double *wk = nullptr;
    int *arr = nullptr;
    if (ksplit > 1 && cs == 0) wk = work.ensure((size_t)ksplit * batch * m * n);
    if (ksplit > 1 && cs > 0) {
      if (ksplit > cs) wk = work.ensure((size_t)(ksplit / cs) * batch * tiles * dg::BM * bn);
      // counters of the last arrivals: zero between launches
      const size_t need = (size_t)batch * tiles * cs;
      if (need > arrived.n) {
        arr = arrived.ensure(std::max<size_t>(need, 4096));
        S2G_CUDA(cudaMemsetAsync(arr, 0, sizeof(int) * arrived.n, s));
      }
      arr = arrived.get();
    }
    const dim3 grid(tiles, batch * ksplit), cluster(1, std::max(cs, 1));
    // the CTAs of a wave share the operand whose tiles change slowest: along n
    // first where A is the larger operand and does not stay in the L2 (65000 x
    // 6000 x 336: with m first A is read anew for every column tile, 11.7 ms in
    // the PT selection of C294H42 against 10.0 ms)
    const int nfast = m > n && (double)m * k * sizeof(double) > 64e6;
#define S2G_DGEMM(TA_, TB_, BN_)                                                              \
  do {                                                                                        \
    bool &ready = smem_set[TA_][TB_][BN_ == 64];                                             \
    if (!ready)                                                                               \
      S2G_CUDA(cudaFuncSetAttribute(k_dgemm<TA_, TB_, BN_>,                                   \
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,              \
                                    dg::smem_bytes<BN_>()));                                  \
    ready = true;                                                                             \
    launch_cluster(k_dgemm<TA_, TB_, BN_>, grid, dg::THREADS, dg::smem_bytes<BN_>(), cluster, \
                   s, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, ksplit,       \
                   kchunk, wk, tri, nfast, cs, arr, sc);                                      \
  } while (0)
    if (bn == 32) {
      if (!ta && !tb) S2G_DGEMM(false, false, 32);
      else if (!ta && tb) S2G_DGEMM(false, true, 32);
      else if (ta && !tb) S2G_DGEMM(true, false, 32);
      else S2G_DGEMM(true, true, 32);
    } else {
      if (!ta && !tb) S2G_DGEMM(false, false, 64);
      else if (!ta && tb) S2G_DGEMM(false, true, 64);
      else if (ta && !tb) S2G_DGEMM(true, false, 64);
      else S2G_DGEMM(true, true, 64);
    }
#undef S2G_DGEMM
    ++launches;
    if (ksplit > 1 && cs == 0) {
      const int64_t total = (int64_t)m * n * batch;
      const int g = (int)std::min<int64_t>(div_up(total, kReduceThreads), (int64_t)nsm * 32);
      S2G_LAUNCH(k_dgemm_reduce, g, kReduceThreads, 0, s, m, n, batch, ksplit, alpha, wk, beta, C,
                 ldc, sC, sc, tb);
      ++launches;
    }
  }
};

}  // namespace std2g
