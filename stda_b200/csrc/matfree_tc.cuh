// Matrix-free J X on the tensor cores (mixed form of the Davidson products).
//
// Same factorisation as matfree.cuh (J X = C_v^T P^A_oo (C_v X^T), per atom A),
// but every GEMM is the split-BF16 tcgen05 contraction of tc_gemm.cuh:
//   G1: Z[R, (r,j)]      = sum_b  Cv[R, b] * XbT[(r,j), b]        (one launch)
//   G2: T_A[(s,r), i]    = sum_j  Z_A[(s,r), j] * P^A[i, j]       (batched over atoms)
//   G3: Y[(i,r), a]      = sum_R  Tt[(i,r), R] * Cv[R, a]^T       (one launch)
// R runs over the padded AO slots (atom A, slot s), j/i over occupied and a/b
// over virtual MOs of the active window, r over the vectors of the block.  G1's
// epilogue writes the BF16 pair that G2 reads, row (R, r) after row; a tiled
// transpose writes G3's operand.  (With G1 the other way round, FP32 Z, a
// transpose and zeroed paddings between the two cost as much as the product itself:
// 0.24 + 0.24 ms per 50 vectors of C384H48, 48 of 105 us per 15 of a 200-atom chain.)  The K part (p_u . sum_v q_v X_v) is two thin
// FP64 GEMMs.  The exchange-type products K_x X ((ib|ja), the velocity
// correction and A +- B) follow the same pattern with C_o and P^A_ov:
//   G1x: Z2[R, (r,b)] = sum_j Co[R, j] X[(r,b), j],
//   G2x: U_A[(s,r), i] = sum_b Z2_A[(s,r), b] P^A_ov[i, b],
// and U joins T before G3.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace std2g {

inline int ld64(int64_t x) { return (int)((x + 63) / 64 * 64); }
inline int ld4(int64_t x) { return (int)((x + 3) / 4 * 4); }

__device__ __forceinline__ void split_store(__nv_bfloat16 *hi, __nv_bfloat16 *lo, int64_t o,
                                            double x) {
  __nv_bfloat16 h = __double2bfloat16(x);
  hi[o] = h;
  lo[o] = __double2bfloat16(x - (double)__bfloat162float(h));
}

// Loewdin MO operands: mode 0: out[R*Kp + b] = Cv[R, b] (R < nrow = AO slots);
// mode 1: out[a*Kp + R] = Cv[R, a] (a < nrow = nv); mode 2: out[R*Kp + j] =
// Co[R, j] (R < nrow = AO slots, j < no).  Zero beyond the data.
__global__ void k_tcs_clow(__nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                           const double *__restrict__ Clow, int nao, const int *__restrict__ slot,
                           int rows, int no, int nv, int nrow, int Kp, int mode) {
  int64_t total = (int64_t)nrow * Kp;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int row = (int)(t / Kp), k = (int)(t - (int64_t)row * Kp);
    int R = mode == 1 ? k : row, c = mode == 1 ? row : k;
    double x = 0.0;
    const int ncol = mode == 2 ? no : nv, col0 = mode == 2 ? 0 : no;
    if (R < rows && c < ncol) {
      int ao = slot[R];
      if (ao >= 0) x = Clow[ao + (int64_t)nao * (col0 + c)];
    }
    split_store(hi, lo, t, x);
  }
}

// Atom-major rows of a pair tensor: out[A*n1*K2 + i*K2 + j] = P[A + N*(i*n2 + j)]
// (i < n1, j < n2; P^A_oo with n1 = n2 = no, P^A_ov with n1 = no, n2 = nv;
// padding columns are left as they are).  Tiled over (atoms, pairs).
__global__ void k_tcs_pairs(__nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                            const double *__restrict__ P, int N, int n1, int n2, int K2) {
  __shared__ double tile[32][33];
  const int64_t np = (int64_t)n1 * n2;
  const int A0 = blockIdx.x * 32, tx = threadIdx.x;
  for (int64_t p0 = (int64_t)blockIdx.y * 32; p0 < np; p0 += (int64_t)gridDim.y * 32) {
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
      int64_t p = p0 + ty;
      int A = A0 + tx;
      if (A < N && p < np) tile[ty][tx] = P[A + (int64_t)N * p];
    }
    __syncthreads();
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
      int A = A0 + ty;
      int64_t p = p0 + tx;
      if (A < N && p < np) {
        int64_t i = p / n2, j = p - i * n2;
        split_store(hi, lo, (int64_t)A * n1 * K2 + i * K2 + j, tile[tx][ty]);
      }
    }
    __syncthreads();
  }
}

// out[(g + ng*r)*Kp + f] = X[u + nci*r] with u = pos[f + nf*g], zero where there is no
// CSF, for f >= nf and for g >= nrow (ng: rows per vector, Kp a multiple of 8).  Eight
// elements per thread; one pass instead of two memsets and a scatter.
__global__ void k_tcs_box(__nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                          const double *__restrict__ X, const int *__restrict__ pos, int nci,
                          int nf, int nrow, int ng, int Kp, int m) {
  const int64_t total = (int64_t)(Kp / 8) * ng * m;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t / (Kp / 8);
    const int f0 = (int)(t - c * (Kp / 8)) * 8, r = (int)(c / ng), g = (int)(c - (int64_t)r * ng);
    __align__(16) __nv_bfloat16 h[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int f = f0 + e;
      const int u = f < nf && g < nrow ? pos[f + (int64_t)nf * g] : -1;
      const double x = u >= 0 ? X[u + (int64_t)nci * r] : 0.0;
      h[e] = __double2bfloat16(x);
      l[e] = __double2bfloat16(x - (double)__bfloat162float(h[e]));
    }
    *reinterpret_cast<uint4 *>(hi + c * Kp + f0) = *reinterpret_cast<const uint4 *>(h);
    *reinterpret_cast<uint4 *>(lo + c * Kp + f0) = *reinterpret_cast<const uint4 *>(l);
  }
}

// f T + fU U, both [(R*m + r)*ldo + i] (either may be NULL) -> Tt[(i + no*r)*KR + R].
// grid (no/32, rows/32, m), block 32x8; columns R >= rows are left as they are.
__global__ void k_tcs_from_atom(__nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo,
                                const float *__restrict__ T, const float *__restrict__ U,
                                int ldo, int rows, int no, int KR, int m, double f, double fU) {
  __shared__ float tile[32][33];
  const int i0 = blockIdx.x * 32, R0 = blockIdx.y * 32, r = blockIdx.z, tx = threadIdx.x;
  for (int ty = threadIdx.y; ty < 32; ty += 8) {
    int R = R0 + ty, i = i0 + tx;
    if (i < no && R < rows) {
      const int64_t o = ((int64_t)R * m + r) * ldo + i;
      float v = 0.f;
      if (T) v += (float)f * T[o];
      if (U) v += (float)fU * U[o];
      tile[ty][tx] = v;
    }
  }
  __syncthreads();
  for (int ty = threadIdx.y; ty < 32; ty += 8) {
    int i = i0 + ty, R = R0 + tx;
    if (i < no && R < rows)
      split_store(hi, lo, ((int64_t)i + (int64_t)no * r) * KR + R, (double)tile[tx][ty]);
  }
}

// out[u + nci*r] += Y[(i_u + no*r)*ldv + a_u] + diag[u] X[u + nci*r] (diag may be NULL)
__global__ void k_tcs_gather(double *__restrict__ out, const float *__restrict__ Y, int ldv,
                             const int *__restrict__ ci, const int *__restrict__ ca, int nci,
                             int no, int m, const double *__restrict__ X,
                             const double *__restrict__ diag) {
  int64_t total = (int64_t)nci * m;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(t / nci), u = (int)(t - (int64_t)r * nci);
    double v = out[t] + (double)Y[((int64_t)ci[u] + (int64_t)no * r) * ldv + ca[u]];
    if (diag) v = fma(diag[u], X[t], v);
    out[t] = v;
  }
}

// A second stream with its own cuBLAS handle, on which the FP64 exchange
// part of the product runs concurrently with the tensor-core Coulomb part.
struct SideStream {
  cudaStream_t s = nullptr;
  cublasHandle_t h = nullptr;
  Dgemm dg;   // FP64 products on this stream (own split-K workspace)
  bool lib_fp64 = false;   // those products through cuBLAS (STD2G_FLAG_LIBRARY_FP64)
  cudaEvent_t fork = nullptr, join = nullptr;
  void init() {
    if (s) return;
    S2G_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    S2G_CUBLAS(cublasCreate(&h));
    S2G_CUBLAS(cublasSetStream(h, s));
    if (lib_fp64) dg.lib = h;
    S2G_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    S2G_CUDA(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
  }
  ~SideStream() {
    if (h) cublasDestroy(h);
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    if (s) cudaStreamDestroy(s);
  }
};

struct MatFreeTc {
  int N = 0, maxa = 0, no = 0, nv = 0, nci = 0, rows = 0;
  int Kv = 0, Ko = 0, KR = 0;
  const double *Qs = nullptr, *Ps = nullptr;   // FP64 [csf][atom] charges for the K part
  const int *ci = nullptr, *ca = nullptr;
  TcGemm tc;
  DBuf<__nv_bfloat16> cvt_h, cvt_l, cv2_h, cv2_l, poo_h, poo_l;
  DBuf<__nv_bfloat16> xb_h, xb_l, zt_h, zt_l, tt_h, tt_l;
  DBuf<float> T, Y;
  DBuf<int> pos;   // positions of the CSFs (k_mf_positions)
  // exchange chain (K_x X, the (ib|ja) products): C_o rows, P^A_ov rows
  bool has_x = false;
  DBuf<__nv_bfloat16> cot_h, cot_l, pov_h, pov_l, xv_h, xv_l, z2t_h, z2t_l;
  DBuf<float> U;
  DBuf<double> G;
  SideStream side;
};

// Operands fixed for the solve: Cv in both K-major orientations, P^A_oo rows.
inline void mftc_setup(MatFreeTc &w, cudaStream_t s, const double *Clow, int nao,
                       const int *slot, const double *Poo, const double *Pia = nullptr) {
  w.rows = w.N * w.maxa;
  w.Kv = ld64(w.nv);
  w.Ko = ld64(w.no);
  w.KR = ld64(w.rows);
  const int g = 148 * 16;
  S2G_LAUNCH(k_tcs_clow, g, 256, 0, s, w.cvt_h.ensure((size_t)w.rows * w.Kv),
             w.cvt_l.ensure((size_t)w.rows * w.Kv), Clow, nao, slot, w.rows, w.no, w.nv, w.rows,
             w.Kv, 0);
  S2G_LAUNCH(k_tcs_clow, g, 256, 0, s, w.cv2_h.ensure((size_t)w.nv * w.KR),
             w.cv2_l.ensure((size_t)w.nv * w.KR), Clow, nao, slot, w.rows, w.no, w.nv, w.nv, w.KR,
             1);
  const size_t np = (size_t)w.N * w.no * w.Ko;
  __nv_bfloat16 *ph = w.poo_h.ensure(np), *pl = w.poo_l.ensure(np);
  S2G_LAUNCH(k_tcs_pairs,
             dim3((unsigned)div_up(w.N, 32),
                  (unsigned)std::min<int64_t>(div_up((int64_t)w.no * w.no, 32), 65535)),
             dim3(32, 8), 0, s, ph, pl, Poo, w.N, w.no, w.no, w.Ko);
  int *pos = w.pos.ensure((size_t)2 * w.no * w.nv);
  S2G_CUDA(cudaMemsetAsync(pos, 0xff, sizeof(int) * 2 * w.no * w.nv, s));
  S2G_LAUNCH(k_mf_positions, (int)div_up(w.nci, 256), 256, 0, s, pos, w.ci, w.ca, w.nci, w.no,
             w.nv);
  w.has_x = Pia != nullptr;
  if (w.has_x) {
    S2G_LAUNCH(k_tcs_clow, g, 256, 0, s, w.cot_h.ensure((size_t)w.rows * w.Ko),
               w.cot_l.ensure((size_t)w.rows * w.Ko), Clow, nao, slot, w.rows, w.no, w.nv, w.rows,
               w.Ko, 2);
    const size_t nq = (size_t)w.N * w.no * w.Kv;
    __nv_bfloat16 *qh = w.pov_h.ensure(nq), *ql = w.pov_l.ensure(nq);
    S2G_LAUNCH(k_tcs_pairs,
               dim3((unsigned)div_up(w.N, 32),
                    (unsigned)std::min<int64_t>(div_up((int64_t)w.no * w.nv, 32), 65535)),
               dim3(32, 8), 0, s, qh, ql, Pia, w.N, w.no, w.nv, w.Kv);
  }
}

// out (nci x m, FP64) = cK (K X) + cJ (J X) + cX (K_x X) + diag o X
// (cX != 0 needs the exchange operands of mftc_setup(..., Pia))
inline void mftc_apply(MatFreeTc &w, cudaStream_t s, const double *X, int m,
                       double *out, double cK, double cJ, double cX, const double *diag) {
  const int N = w.N, no = w.no, nv = w.nv, nci = w.nci, rows = w.rows, maxa = w.maxa;
  const int g = 148 * 8;
  if (cX != 0.0 && !w.has_x) throw Error{STD2G_ESTATE, "mftc_apply: exchange operands not set up"};
  // K part, out = cK Ps^T (Qs X), in FP64 on the side stream
  const bool side = cK != 0.0;
  if (side) {
    w.side.init();
    S2G_CUDA(cudaEventRecord(w.side.fork, s));
    S2G_CUDA(cudaStreamWaitEvent(w.side.s, w.side.fork, 0));
    double *G = w.G.ensure((size_t)N * m);
    const double one = 1.0, zero = 0.0, ck = cK;
    w.side.dg.gemm(w.side.s, CUBLAS_OP_N, CUBLAS_OP_N, N, m, nci, &one, w.Qs, N, X, nci, &zero,
                   G, N);
    w.side.dg.gemm(w.side.s, CUBLAS_OP_T, CUBLAS_OP_N, nci, m, N, &ck, w.Ps, N, G, N, &zero, out,
                   nci);
    S2G_CUDA(cudaEventRecord(w.side.join, w.side.s));
  } else {
    S2G_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * nci * m, s));
  }
  if (cJ != 0.0 || cX != 0.0) {
    const int64_t mo = (int64_t)no * m, mz = (int64_t)maxa * m;
    const int ldo = ld4(no), ldv = ld4(nv), Zo = ld8(no), Zv = ld8(nv);
    const dim3 tb(32, 8);
    float *T = nullptr, *U = nullptr;
    if (cJ != 0.0) {
      // G1: Z[R, (r,j)] = sum_b Cv[R, b] X_jb^r, j padded to Zo
      const size_t nx = (size_t)m * Zo * w.Kv, nz = (size_t)rows * m * Zo;
      __nv_bfloat16 *xh = w.xb_h.ensure(nx), *xl = w.xb_l.ensure(nx);
      S2G_LAUNCH(k_tcs_box, g, 256, 0, s, xh, xl, X, w.pos.get(), nci, nv, no, Zo, w.Kv, m);
      __nv_bfloat16 *zh = w.zt_h.ensure(nz), *zl = w.zt_l.ensure(nz);
      w.tc.run(s, w.cvt_h.get(), w.cvt_l.get(), w.Kv, xh, xl, w.Kv, rows, m * Zo, nv, zh, zl,
               (int64_t)m * Zo, 2.0 * mo * rows * nv);
      // G2: T_A[(s,r), i] = sum_j Z_A[(s,r), j] P^A_oo[i, j], batched over atoms
      T = w.T.ensure((size_t)N * mz * ldo);
      w.tc.run(s, zh, zl, Zo, w.poo_h.get(), w.poo_l.get(), w.Ko, (int)mz, no, no, T, nullptr, ldo,
               2.0 * mz * no * no, N, true, mz * ldo);
    }
    if (cX != 0.0) {
      // G1x: Z2[R, (r,b)] = sum_j Co[R, j] X_jb^r, b padded to Zv
      const int64_t mv = (int64_t)nv * m;
      const size_t nx = (size_t)m * Zv * w.Ko, nz = (size_t)rows * m * Zv;
      __nv_bfloat16 *xh = w.xv_h.ensure(nx), *xl = w.xv_l.ensure(nx);
      S2G_LAUNCH(k_tcs_box, g, 256, 0, s, xh, xl, X, w.pos.get() + (int64_t)no * nv, nci, no, nv,
                 Zv, w.Ko, m);
      __nv_bfloat16 *zh = w.z2t_h.ensure(nz), *zl = w.z2t_l.ensure(nz);
      w.tc.run(s, w.cot_h.get(), w.cot_l.get(), w.Ko, xh, xl, w.Ko, rows, m * Zv, no, zh, zl,
               (int64_t)m * Zv, 2.0 * mv * rows * no);
      // G2x: U_A[(s,r), i] = sum_b Z2_A[(s,r), b] P^A_ov[i, b], batched over atoms
      U = w.U.ensure((size_t)N * mz * ldo);
      w.tc.run(s, zh, zl, Zv, w.pov_h.get(), w.pov_l.get(), w.Kv, (int)mz, no, nv, U, nullptr, ldo,
               2.0 * mz * no * nv, N, true, mz * ldo);
    }
    // G3 operand: cJ T + cX U back to (i, r) rows; G3: Y[(i,r), a] = sum_R Tt Cv[R, a]
    __nv_bfloat16 *th = w.tt_h.ensure((size_t)mo * w.KR), *tl = w.tt_l.ensure((size_t)mo * w.KR);
    S2G_LAUNCH(k_tcs_from_atom, dim3((unsigned)div_up(no, 32), (unsigned)div_up(rows, 32), (unsigned)m),
               tb, 0, s, th, tl, T, U, ldo, rows, no, w.KR, m, cJ, cX);
    float *Y = w.Y.ensure((size_t)mo * ldv);
    w.tc.run(s, th, tl, w.KR, w.cv2_h.get(), w.cv2_l.get(), w.KR, (int)mo, nv, rows, Y, nullptr,
             ldv, 2.0 * mo * nv * rows);
    if (side) S2G_CUDA(cudaStreamWaitEvent(s, w.side.join, 0));
    S2G_LAUNCH(k_tcs_gather, g, 256, 0, s, out, Y, ldv, w.ci, w.ca, nci, no, m, X, diag);
    w.tc.poll(s);
  } else {
    if (side) S2G_CUDA(cudaStreamWaitEvent(s, w.side.join, 0));
    if (diag) S2G_LAUNCH(k_add_diag, g, 256, 0, s, out, X, diag, nci, m);
  }
}

}  // namespace std2g
