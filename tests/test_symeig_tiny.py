"""The small eigensolver on matrices with couplings whose squares are below the
smallest normal number (the charges of far apart fragments give them).  The
couplings do not count beside the diagonal's rounding, so the bounds are those of
the other matrices: eigenvalues to 1e-11 ||A||, residuals and orthogonality to
1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 40, 130, 300])
@pytest.mark.parametrize("tiny", [1e-139, 1e-150, 1e-155, 1e-159, 1e-161, 1e-200, 1e-299, 1e-305, 5e-324])
def test_tiny_couplings(n, tiny):
    from stda_b200.engine import symeig_check
    rng = np.random.default_rng(n)
    B = rng.choice([-1.0, 1.0], (n, n)) * rng.integers(1, 8, (n, n)) * tiny
    A = np.tril(B, -1) + np.tril(B, -1).T + np.diag(rng.uniform(0.1, 1.0, n))
    k = min(n, 60)
    w, Z, _ = symeig_check(A, k)
    scale = np.abs(A).sum(axis=1).max()
    assert np.abs(w - np.sort(np.diag(A))[:k]).max() <= 1e-11 * scale
    assert np.abs(A @ Z - Z * w[None, :]).max() <= 1e-10 * scale
    assert np.abs(Z.T @ Z - np.eye(k)).max() <= 1e-10
