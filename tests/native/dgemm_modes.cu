// C entries to the forms of the FP64 product that std2g_dgemm_check does not reach
// (symmetric results, two-level columns, grouped members with indexed columns), on
// host arrays of na, nb, nc doubles.  Return an STD2G_* code.  form: 0 as the engine
// picks, 1 splits by wave counts, 2 cuBLAS.
#include <atomic>

#include "../../stda_b200/csrc/dgemm.cuh"

namespace std2g {
std::atomic<int64_t> g_launches{0};
}
using namespace std2g;

namespace {
struct Arrays {
  DBuf<double> A, B, C;
  cudaStream_t s = nullptr;
  Dgemm g;
  Arrays(const double *a, int64_t na, const double *b, int64_t nb, const double *c, int64_t nc) {
    S2G_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    put(A, a, na);
    put(B, b, nb);
    put(C, c, nc);
    int dev = 0;
    S2G_CUDA(cudaGetDevice(&dev));
    S2G_CUDA(cudaDeviceGetAttribute(&g.nsm, cudaDevAttrMultiProcessorCount, dev));
  }
  ~Arrays() { cudaStreamDestroy(s); }
  void put(DBuf<double> &d, const double *h, int64_t n) {
    S2G_CUDA(cudaMemcpyAsync(d.ensure(n), h, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  }
  void get(double *c, int64_t nc) {
    S2G_CUDA(cudaMemcpyAsync(c, C.get(), sizeof(double) * nc, cudaMemcpyDeviceToHost, s));
    S2G_CUDA(cudaStreamSynchronize(s));
  }
};

struct Handle {
  cublasHandle_t b = nullptr;
  ~Handle() {
    if (b) cublasDestroy(b);
  }
};

template <class F>
int code_of(F &&f) {
  try {
    f();
    return STD2G_OK;
  } catch (const Error &e) {
    return e.code;
  }
}
}  // namespace

extern "C" int dg_run(int form, int ta, int tb, int m, int n, int k, double alpha,
                      const double *A, int64_t na, int64_t lda, int64_t sA, const double *B,
                      int64_t nb, int64_t ldb, int64_t sB, double beta, double *C, int64_t nc,
                      int64_t ldc, int64_t sC, int batch, int tri, int len, int64_t colB,
                      int64_t colC) {
  return code_of([&] {
    Arrays x(A, na, B, nb, C, nc);
    x.g.wave_splits = form == 1;
    Handle h;
    if (form == 2) {
      S2G_CUBLAS(cublasCreate(&h.b));
      x.g.lib = h.b;
    }
    x.g.run(x.s, ta != 0, tb != 0, m, n, k, alpha, x.A.get(), lda, sA, x.B.get(), ldb, sB, beta,
            x.C.get(), ldc, sC, batch, tri, DgSplitCols{len, colB, colC});
    if (form == 2 && x.g.launches != 0) throw Error{STD2G_ESTATE, "own kernel"};
    x.get(C, nc);
  });
}

// members p: C[at C0[p]] = alpha op(A[at A0[p]]) op(B) + beta C, columns named by
// bcol / ccol from col0[p] on (col0[p] < 0: plain columns)
extern "C" int dg_grouped(int form, int ta, int tb, int np, const int *M, const int *N, const int *K,
                          double alpha, double beta, const double *A, int64_t na,
                          const int64_t *A0, int64_t lda, const double *B, int64_t nb,
                          const int64_t *B0, int64_t ldb, double *C, int64_t nc,
                          const int64_t *C0, int64_t ldc, const int *bcol, const int *ccol,
                          int ncol, const int64_t *col0) {
  return code_of([&] {
    Arrays x(A, na, B, nb, C, nc);
    Handle h;
    if (form == 2) {
      S2G_CUBLAS(cublasCreate(&h.b));
      x.g.lib = h.b;
    }
    DBuf<int> db, dc;
    S2G_CUDA(cudaMemcpyAsync(db.ensure(ncol), bcol, sizeof(int) * ncol, cudaMemcpyHostToDevice, x.s));
    S2G_CUDA(cudaMemcpyAsync(dc.ensure(ncol), ccol, sizeof(int) * ncol, cudaMemcpyHostToDevice, x.s));
    std::vector<DgProblem> pr(np);
    for (int p = 0; p < np; ++p) {
      DgProblem &d = pr[p];
      d.M = M[p];
      d.N = N[p];
      d.K = K[p];
      d.alpha = alpha;
      d.beta = beta;
      d.A = x.A.get() + A0[p];
      d.B = x.B.get() + B0[p];
      d.C = x.C.get() + C0[p];
      d.lda = lda;
      d.ldb = ldb;
      d.ldc = ldc;
      if (col0[p] >= 0) {
        d.bcol = db.get() + col0[p];
        d.ccol = dc.get() + col0[p];
      }
    }
    x.g.grouped(x.s, ta != 0, tb != 0, pr);
    if (form == 2 && x.g.launches != 0) throw Error{STD2G_ESTATE, "own kernel"};
    x.get(C, nc);
  });
}
