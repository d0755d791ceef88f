"""The small eigensolver at the edges of its blockings (multisection rounds of
8 minors, reflector blocks, row blocks of 32 and the CTA / cluster limits) and
on tridiagonal forms with vanishing couplings, against numpy's eigh:
eigenvalues to 1e-11 ||A||, residuals and orthogonality to 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(A, k):
    from stda_b200.engine import symeig_check
    w, Z, _ = symeig_check(A, k)
    wr = np.linalg.eigvalsh(A)[:k]
    scale = np.abs(A).sum(axis=1).max()
    assert np.abs(w - wr).max() <= 1e-11 * scale
    assert np.abs(A @ Z - Z * w[None, :]).max() <= 1e-10 * scale
    assert np.abs(Z.T @ Z - np.eye(k)).max() <= 1e-10


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 10, 11, 16, 17, 31, 32, 33, 34, 63, 64, 65,
                               95, 96, 97, 127, 128, 129, 160, 191, 192, 193, 255, 256, 257, 319,
                               320])
def test_block_edges(n):
    rng = np.random.default_rng(1000 + n)
    M = rng.standard_normal((n, n))
    _check(0.5 * (M + M.T), n if n < 40 else n // 3)


@pytest.mark.parametrize("n", [5, 40, 130, 300])
@pytest.mark.parametrize("scale", [1.0, 1e-120, 1e120])
def test_decoupled_blocks(n, scale):
    """A diagonal matrix with one dense 3 x 3 block: zero off-diagonals in T."""
    rng = np.random.default_rng(n)
    A = np.diag(np.sort(rng.uniform(-1.0, 1.0, n)) + 1e-3 * np.arange(n))
    B = rng.standard_normal((3, 3))
    A[1:4, 1:4] += 0.1 * (B + B.T)
    _check(scale * A, min(n, 60))
