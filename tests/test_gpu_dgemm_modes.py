"""The FP64 product's symmetric results, two-level columns (both orders of op(B), the
engine's kernel and cuBLAS) and grouped members with indexed columns, at the edges of
their tiles, against numpy on the same addresses: |err| <= 4 eps (k + 8) |A| |B| summed, and everything that is not
addressed is left as it was."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from stda_b200.build import NVCC
    out = str(tmp_path_factory.mktemp("native") / "dgemm_modes.so")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", os.path.join(HERE, "native", "dgemm_modes.cu"), "-o", out,
                    "-lcublas"], check=True)
    return ct.CDLL(out)


def _d(a):
    return a.ctypes.data_as(ct.POINTER(ct.c_double))


def _run(lib, ta, tb, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch=1, tri=0, len_=0,
         colB=0, colC=0, form=0):
    out = C.copy()
    L, D = ct.c_int64, ct.c_double
    code = lib.dg_run(form, ta, tb, m, n, k, D(alpha), _d(A), L(A.size), L(lda), L(sA), _d(B), L(B.size),
                      L(ldb), L(sB), D(beta), _d(out), L(C.size), L(ldc), L(sC), batch, tri, len_, L(colB),
                      L(colC))
    return code, out


def _close(got, ref, mag, k):
    return np.all(np.abs(got - ref) <= 4 * 2.2e-16 * (k + 8) * mag)


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0)])
@pytest.mark.parametrize("n,k", [(1, 3), (31, 40), (64, 16), (65, 300), (220, 220), (518, 97)])
def test_symmetric_result(lib, form, ta, tb, n, k):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, k))
    W = rng.standard_normal(k)
    a, b = G * W, G.T                        # a b is symmetric
    A = np.ascontiguousarray(a if ta else a.T).ravel()    # column-major op(A)
    B = np.ascontiguousarray(b.T).ravel()
    code, out = _run(lib, ta, tb, n, n, k, 1.5, A, k if ta else n, 0, B, k, 0, 0.0,
                     np.full(n * n, np.nan), n, 0, tri=-1, form=form)
    assert code == 0
    out = out.reshape(n, n)
    if form == 0:
        assert np.array_equal(out, out.T)
    assert _close(out, 1.5 * a @ b, 1.5 * np.abs(a) @ np.abs(b), k)


def test_symmetric_result_refused_with_wave_splits(lib):
    """Split sums in a second launch would add tiles that were never formed."""
    n = 300
    A = np.eye(n).ravel()
    code, _ = _run(lib, 0, 0, n, n, n, 1.0, A, n, 0, A, n, 0, 0.0, A, n, 0, tri=-1, form=1)
    assert code == 1


@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("m,k,len_,groups,batch", [(5, 3, 1, 1, 2), (64, 16, 4, 15, 3), (65, 130, 9, 8, 4),
                                                   (129, 700, 5, 26, 2), (90, 90, 9, 60, 7)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_two_level_columns(lib, tb, form, m, k, len_, groups, batch, beta):
    rng = np.random.default_rng(m + k)
    lda, n = m + 3, len_ * groups
    sA = lda * k
    A = rng.standard_normal(sA * batch)
    # group g, batch member q: in an array whose leading dimension holds all members
    rows = len_ * batch + 2
    if tb:
        ldb, sB, colB = rows, len_, rows * k + 5
        ldc, sC, colC = rows, len_, rows * m + 7
    else:
        ldb, ldc = k + 1, m + 2
        sB, colB = ldb * len_, ldb * rows
        sC, colC = ldc * len_, ldc * rows
    B = rng.standard_normal(colB * groups)
    C = rng.standard_normal(colC * groups)
    code, out = _run(lib, 0, tb, m, n, k, -1.5, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, 0, len_,
                     colB, colC, form)
    assert code == 0
    ref, mag = C.copy(), np.zeros_like(C)
    i, kk = np.arange(m), np.arange(k)
    for q in range(batch):
        a = A[q * sA + i[:, None] + lda * kk[None, :]]
        for g in range(groups):
            for c in range(len_):
                b = B[q * sB + g * colB + (c + ldb * kk if tb else c * ldb + kk)]
                at = q * sC + g * colC + (c + ldc * i if tb else c * ldc + i)
                ref[at] = -1.5 * (a @ b) + beta * C[at]
                mag[at] = 1.5 * (np.abs(a) @ np.abs(b)) + np.abs(C[at])
    assert _close(out, ref, mag, k)


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("M,N,K", [([7, 70], [3, 33], [5, 20]), ([64] * 9, [1, 2, 31, 32, 33, 63, 64, 65, 7], [141] * 9),
                                   ([588] * 45, [64] * 45, [48] * 45)])
def test_grouped_indexed_columns(lib, form, M, N, K):
    """Each member adds to the columns that its list names; one launch, 32- and
    64-wide tiles."""
    rng = np.random.default_rng(len(M))
    np_, ld, kmax = len(M), max(M), max(K)
    ncol = sum(N)
    A = rng.standard_normal(kmax * ld * np_)            # op(A) = A^T: K x M each
    nbcol = ncol + 11
    B = rng.standard_normal(kmax * nbcol)
    bcol = rng.integers(0, nbcol, ncol).astype(np.int32)
    ccol = rng.permutation(ncol + 5)[:ncol].astype(np.int32)
    C = rng.standard_normal(ld * (ncol + 5))
    A0 = np.arange(np_, dtype=np.int64) * kmax * ld
    zero = np.zeros(np_, dtype=np.int64)
    col0 = np.concatenate([[0], np.cumsum(N)[:-1]]).astype(np.int64)
    i32 = lambda v: np.asarray(v, dtype=np.int32)  # noqa: E731
    p = lambda v, t: v.ctypes.data_as(ct.POINTER(t))  # noqa: E731
    Mi, Ni, Ki = i32(M), i32(N), i32(K)
    out, L, D = C.copy(), ct.c_int64, ct.c_double
    code = lib.dg_grouped(form, 1, 0, np_, p(Mi, ct.c_int), p(Ni, ct.c_int), p(Ki, ct.c_int), D(-1.0), D(1.0), _d(A),
                          L(A.size), p(A0, L), L(kmax), _d(B), L(B.size), p(zero, L), L(kmax), _d(out),
                          L(C.size), p(zero, L), L(ld), p(bcol, ct.c_int), p(ccol, ct.c_int), ncol, p(col0, L))
    assert code == 0
    ref, mag = C.reshape(-1, ld).copy(), np.zeros((ncol + 5, ld))
    Bm = B.reshape(nbcol, kmax)
    for q in range(np_):
        a = A[A0[q]:A0[q] + kmax * ld].reshape(ld, kmax)[:M[q], :K[q]]
        for c in range(N[q]):
            b, at = Bm[bcol[col0[q] + c], :K[q]], ccol[col0[q] + c]
            ref[at, :M[q]] -= a @ b
            mag[at, :M[q]] = np.abs(a) @ np.abs(b) + np.abs(C.reshape(-1, ld)[at, :M[q]])
    assert _close(out.reshape(-1, ld), ref, mag, kmax)
