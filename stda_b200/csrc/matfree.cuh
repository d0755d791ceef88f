// Matrix-free products with the sTDA / sTD-DFT matrices.
//
// The reference builds A (rtdamat, stda.f:2010-2056), A+B / A-B (rrpamat,
// stda.f:1870-2004) and 0.5 B (rtdacorr, apbtrafo.f:580-643) element by
// element, each element being a gathered dot product over atoms:
//   (ia|jb) = p_ia . q_jb    (gamma^K)
//   (ij|ab) = p_ij . q_ab    (gamma^J)
//   (ib|ja) = p_ib . q_ja    (gamma^K)
// Here only products M X with blocks of vectors X are formed, never M itself.
// With the Loewdin MOs C (q_pq^A = sum_{k in A} C_kp C_kq) the three couplings
// factor into dense GEMMs:
//   K X   : g = sum_v q_v X_v (N x m), then p_u . g               -- 2 GEMMs
//   J X   : Z = C_v X^T  ->  T_A = P^A_oo Z_A  ->  C_v^T T      -- 3 GEMMs
//   Kx X  : Z = C_o X    ->  U_A = P^A_ov Z_A  ->  C_v^T U      -- 3 GEMMs
// where A runs over atoms, Z_A / T_A / U_A hold the rows of the AOs on atom A
// (padded to `maxa` slots per atom) and P^A are gamma-contracted charges in
// atom-major layout.  Every term of the element-wise definition is included
// (the diagonal ones too), so A X only needs the correction
// ed - (ak K_uu - J_uu) on the diagonal.
#pragma once

#include "common.cuh"
#include "dgemm.cuh"

namespace std2g {

// Leading dimensions are padded to multiples of 8 elements so that every GEMM
// operand is 16-byte aligned (required for the tensor-core GEMM paths).
inline int ld8(int64_t x) { return (int)((x + 7) / 8 * 8); }

// pos[b + nv*j] = pos[no*nv + j + no*b] = the CSF (j, b), -1 where there is none (both
// tables filled with -1 before)
__global__ void k_mf_positions(int *__restrict__ pos, const int *__restrict__ ci,
                               const int *__restrict__ ca, int nci, int no, int nv) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= nci) return;
  pos[ca[u] + (int64_t)nv * ci[u]] = u;
  pos[(int64_t)no * nv + ci[u] + (int64_t)no * ca[u]] = u;
}

// box[f + ld*(g + ns*r)] = X[u + nci*r] with u = pos[f + nf*g], zero where there is no
// CSF and for f >= nf: one pass over the box instead of a memset and a scatter
__global__ void k_mf_box(double *__restrict__ box, const double *__restrict__ X,
                         const int *__restrict__ pos, int nci, int nf, int ns, int ld, int m) {
  const int64_t total = (int64_t)ld * ns * m;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t / ld;
    const int f = (int)(t - c * ld), r = (int)(c / ns), g = (int)(c - (int64_t)r * ns);
    const int u = f < nf ? pos[f + (int64_t)nf * g] : -1;
    box[t] = u >= 0 ? X[u + (int64_t)nci * r] : 0.0;
  }
}

// out = (have ? out : 0) + box[a_u + ldv*(i_u + no*r)] + diag[u] X  (diag may be NULL)
__global__ void k_mf_gather(double *__restrict__ out, const double *__restrict__ box,
                            const int *__restrict__ ci, const int *__restrict__ ca, int nci, int no,
                            int ldv, int m, int have, const double *__restrict__ X,
                            const double *__restrict__ diag) {
  int64_t total = (int64_t)nci * m;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int r = (int)(t / nci), u = (int)(t - (int64_t)r * nci);
    double v = have ? out[t] : 0.0;
    v += box[ca[u] + (int64_t)ldv * (ci[u] + (int64_t)no * r)];
    if (diag) v = fma(diag[u], X[t], v);
    out[t] = v;
  }
}

// dst[A*ld1*n2 + i + ld1*b] = src[A + N*(i*n2 + b)]: [pair (i,b)][atom] -> per atom
// an n1 x n2 column-major matrix with leading dimension ld1.  Tiled; grid
// (N/32, <=65535), block 32x8.
template <typename T>
__global__ void k_pair_to_atom_major(T *__restrict__ dst, const double *__restrict__ src, int N,
                                     int n1, int n2, int ld1) {
  __shared__ double tile[32][33];
  const int64_t np = (int64_t)n1 * n2;
  const int A0 = blockIdx.x * 32;
  const int tx = threadIdx.x;
  for (int64_t p0 = (int64_t)blockIdx.y * 32; p0 < np; p0 += (int64_t)gridDim.y * 32) {
    // p0: pair index i + n1*b of the tile's first column
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
      int64_t pp = p0 + ty;
      int A = A0 + tx;
      if (A < N && pp < np) {
        int64_t b = pp / n1, i = pp - b * n1;
        tile[ty][tx] = src[A + (int64_t)N * (i * n2 + b)];
      }
    }
    __syncthreads();
    for (int ty = threadIdx.y; ty < 32; ty += 8) {
      int A = A0 + ty;
      int64_t pp = p0 + tx;
      if (A < N && pp < np) {
        int64_t b = pp / n1, i = pp - b * n1;
        dst[(int64_t)A * ld1 * n2 + i + (int64_t)ld1 * b] = (T)tile[tx][ty];
      }
    }
    __syncthreads();
  }
}

// out[t] += d[t % n] * X[t]
__global__ void k_add_diag(double *__restrict__ out, const double *__restrict__ X,
                           const double *__restrict__ d, int n, int m) {
  int64_t total = (int64_t)n * m;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x)
    out[t] += d[t % n] * X[t];
}

// padded AO rows: out[(A*maxa+s) + ldr*c] = C[slot_ao[A*maxa+s] + nao*(c0+c)] or 0
// for rows < ldr (rows beyond N*maxa are zero)
template <typename T>
__global__ void k_mf_pad_rows(T *__restrict__ out, const double *__restrict__ C, int nao,
                              const int *__restrict__ slot_ao, int rows, int ldr, int c0,
                              int ncol) {
  int64_t total = (int64_t)ldr * ncol;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int c = (int)(t / ldr), r = (int)(t - (int64_t)c * ldr);
    int k = r < rows ? slot_ao[r] : -1;
    out[t] = k >= 0 ? (T)C[k + (int64_t)nao * (c0 + c)] : (T)0;
  }
}

// diagonal correction for A: dA[u] = ed[u] - (ak*ek[u] - (ii|aa))
__global__ void k_mf_diag(double *__restrict__ dA, const double *__restrict__ ed,
                          const double *__restrict__ ekd, const double *__restrict__ uci,
                          const int *__restrict__ ci, const int *__restrict__ ca, int nci, int nv,
                          double ak) {
  int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= nci) return;
  double jd = uci[ca[u] + (int64_t)nv * ci[u]];
  dA[u] = ed[u] - (ak * ekd[u] - jd);
}

struct MatFree {
  int N = 0, maxa = 0, no = 0, nv = 0, nci = 0, nao = 0;
  Dgemm *dg = nullptr;
  DBuf<double> dA;
  const int *ci = nullptr, *ca = nullptr;
  // operands fixed for a solve: Loewdin MO rows per AO slot, P^A in atom-major
  // layout, the charges of the CSFs (the solve's arrays), CSF positions
  DBuf<double> CvP, CoP, PooA, PovA;
  const double *Qs = nullptr, *Ps = nullptr;
  DBuf<int> pos;
  // work arrays
  DBuf<double> box, Z, Tacc, G;
};

// Set up the operands from the arrays of the solve (once per solve; mf.ci, mf.ca
// and the dimensions set before).
inline void mf_setup_ops(MatFree &mf, cudaStream_t s, const double *Clow, const int *slot_ao,
                         const double *Poo, const double *Pia, const double *Qs, const double *Ps,
                         bool need_ov) {
  const int N = mf.N, rows = N * mf.maxa, no = mf.no, nv = mf.nv, nao = mf.nao;
  const int lr = ld8(rows), lo = ld8(no);
  const int grid = 148 * 16;
  S2G_LAUNCH(k_mf_pad_rows<double>, grid, 256, 0, s, mf.CvP.ensure((size_t)lr * nv), Clow, nao,
             slot_ao, rows, lr, no, nv);
  S2G_LAUNCH(k_mf_pad_rows<double>, grid, 256, 0, s, mf.CoP.ensure((size_t)lr * no), Clow, nao,
             slot_ao, rows, lr, 0, no);
  const dim3 tb(32, 8);
  S2G_LAUNCH(k_pair_to_atom_major<double>,
             dim3((unsigned)div_up(N, 32), (unsigned)std::min<int64_t>(div_up((int64_t)no * no, 32), 65535)),
             tb, 0, s, mf.PooA.ensure((size_t)N * lo * no), Poo, N, no, no, lo);
  if (need_ov)
    S2G_LAUNCH(k_pair_to_atom_major<double>,
               dim3((unsigned)div_up(N, 32), (unsigned)std::min<int64_t>(div_up((int64_t)no * nv, 32), 65535)),
               tb, 0, s, mf.PovA.ensure((size_t)N * lo * nv), Pia, N, no, nv, lo);
  mf.Qs = Qs;
  mf.Ps = Ps;
  int *pos = mf.pos.ensure((size_t)2 * no * nv);
  S2G_CUDA(cudaMemsetAsync(pos, 0xff, sizeof(int) * 2 * no * nv, s));
  S2G_LAUNCH(k_mf_positions, (int)div_up(mf.nci, 256), 256, 0, s, pos, mf.ci, mf.ca, mf.nci, no, nv);
}

// out (nci x m) = cK (K X) + cJ (J X) + cX (Kx X) + diag o X  (diag may be NULL).
// Seven launches for A X: a block of 25 vectors of a 60-atom molecule is bound by
// their latency.  The atoms' products work in place in an array over all AOs
// (DgSplitCols), where two transposes moved both arrays.  That array is [AO][orbital],
// with one product per vector around it, so that every load and store of the atoms'
// products is contiguous.  Where the sums are to be split as before (wave_splits) it is
// [orbital][AO] over all vectors at once, whose runs are the 4 to 9 AOs of an atom: 336
// products 432 x 248 x 432 take 2.10 ms on those and 1.2 on contiguous ones, alpha(w) of
// 57 atoms 10.1 and 9.05, of a 200-atom chain 34.3 and 32.9 ms, 20 and 61 atoms the same.
inline void mf_apply(MatFree &mf, cudaStream_t s, const double *X, int m, double *out, double cK,
                     double cJ, double cX, const double *diag) {
  const int N = mf.N, maxa = mf.maxa, no = mf.no, nv = mf.nv, nci = mf.nci;
  const int rows = N * maxa, lr = ld8(rows), lo = ld8(no), lv = ld8(nv);
  const int grid = 148 * 8;
  Dgemm &dg = *mf.dg;
  const bool box_part = cJ != 0.0 || cX != 0.0;
  if (cK != 0.0) {
    // K part: G = Q_S X (N x m); out = cK P_S^T G
    double *G = mf.G.ensure((size_t)N * m);
    dg.run(s, false, false, N, m, nci, 1.0, mf.Qs, N, 0, X, nci, 0, 0.0, G, N, 0);
    dg.run(s, true, false, nci, m, N, cK, mf.Ps, N, 0, G, N, 0, 0.0, out, nci, 0);
  } else if (!box_part) {
    S2G_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * nci * m, s));
  }
  if (box_part) {
    double *box = mf.box.ensure((size_t)(std::max((int64_t)lv * no, (int64_t)lo * nv) * m));
    double *Z = mf.Z.ensure((size_t)std::max((int64_t)lr * std::max(no, nv),
                                             (int64_t)rows * std::max(lo, lv)) * m);
    double *Tacc = mf.Tacc.ensure((size_t)std::max((int64_t)lr * no, (int64_t)rows * lo) * m);
    const bool by_ao = !dg.wave_splits;
    const int64_t so = (int64_t)(by_ao ? rows : lr) * (by_ao ? lo : no);   // one vector of Tacc
    double beta = 0.0;
    if (cJ != 0.0) {
      S2G_LAUNCH(k_mf_box, grid, 256, 0, s, box, X, mf.pos.get(), nci, nv, no, lv, m);
      if (by_ao) {
        // Z[j + lo*(R + rows*r)] = sum_b X[(j,b),r] CvP[R,b], R = (A, s)
        dg.run(s, true, true, no, rows, nv, 1.0, box, lv, (int64_t)lv * no, mf.CvP.get(), lr, 0, 0.0,
               Z, lo, so, m);
        // atom A: Tacc[i,(s,r)] = cJ sum_j P^A_oo[i,j] Z[j,(s,r)]
        dg.run(s, false, false, no, maxa * m, no, cJ, mf.PooA.get(), lo, (int64_t)lo * no, Z, lo,
               (int64_t)lo * maxa, 0.0, Tacc, lo, (int64_t)lo * maxa, N, 0,
               DgSplitCols{maxa, so, so});
      } else {
        // Z = CvP (rows x nv) * XbT (nv x no*m), XbT[b + lv*(j + no*r)]
        dg.run(s, false, false, rows, no * m, nv, 1.0, mf.CvP.get(), lr, 0, box, lv, 0, 0.0, Z, lr, 0);
        // atom A: Tacc[(s,i,r)] = cJ sum_j P^A_oo[i,j] Z[(s,j,r)], AO slots s of A
        dg.run(s, false, true, no, maxa * m, no, cJ, mf.PooA.get(), lo, (int64_t)lo * no, Z, lr, maxa,
               0.0, Tacc, lr, maxa, N, 0, DgSplitCols{maxa, so, so});
      }
      beta = 1.0;
    }
    if (cX != 0.0) {
      S2G_LAUNCH(k_mf_box, grid, 256, 0, s, box, X, mf.pos.get() + (int64_t)no * nv, nci, no, nv, lo,
                 m);
      if (by_ao) {
        // Z[b + lv*(R + rows*r)] = sum_j X[(j,b),r] CoP[R,j]
        const int64_t sv = (int64_t)rows * lv;
        dg.run(s, true, true, nv, rows, no, 1.0, box, lo, (int64_t)lo * nv, mf.CoP.get(), lr, 0, 0.0,
               Z, lv, sv, m);
        // atom A: Tacc[i,(s,r)] += cX sum_b P^A_ov[i,b] Z[b,(s,r)]
        dg.run(s, false, false, no, maxa * m, nv, cX, mf.PovA.get(), lo, (int64_t)lo * nv, Z, lv,
               (int64_t)lv * maxa, beta, Tacc, lo, (int64_t)lo * maxa, N, 0,
               DgSplitCols{maxa, sv, so});
      } else {
        // Z = CoP (rows x no) * Xb (no x nv*m), Xb[j + lo*(b + nv*r)]
        dg.run(s, false, false, rows, nv * m, no, 1.0, mf.CoP.get(), lr, 0, box, lo, 0, 0.0, Z, lr, 0);
        // atom A: Tacc[(s,i,r)] += cX sum_b P^A_ov[i,b] Z[(s,b,r)]
        dg.run(s, false, true, no, maxa * m, nv, cX, mf.PovA.get(), lo, (int64_t)lo * nv, Z, lr, maxa,
               beta, Tacc, lr, maxa, N, 0, DgSplitCols{maxa, (int64_t)lr * nv, so});
      }
    }
    // box[a + lv*(i + no*r)] = CvP^T (nv x rows) * Tacc (rows x no*m)
    if (by_ao)
      dg.run(s, true, true, nv, no, rows, 1.0, mf.CvP.get(), lr, 0, Tacc, lo, so, 0.0, box, lv,
             (int64_t)lv * no, m);
    else
      dg.run(s, true, false, nv, no * m, rows, 1.0, mf.CvP.get(), lr, 0, Tacc, lr, 0, 0.0, box, lv, 0);
    S2G_LAUNCH(k_mf_gather, grid, 256, 0, s, out, box, mf.ci, mf.ca, nci, no, lv, m, cK != 0.0, X,
               diag);
  } else if (diag) {
    S2G_LAUNCH(k_add_diag, grid, 256, 0, s, out, X, diag, nci, m);
  }
}

}  // namespace std2g
