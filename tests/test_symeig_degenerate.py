"""The small eigensolver on eigenvalues of high multiplicity whose tridiagonal form
falls apart (copies of one block, as non-interacting equal molecules give): the
vectors of a multiplet have to come out independent.  Against numpy's eigh with
the bounds of the other matrices: eigenvalues to 1e-11 ||A||, residuals and
orthogonality to 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,block", [(40, 1), (40, 2), (100, 2), (320, 1), (320, 2), (320, 4), (315, 5)])
def test_copies_of_a_block(n, block):
    from stda_b200.engine import symeig_check
    rng = np.random.default_rng(block)
    B = rng.standard_normal((block, block))
    A = np.kron(np.eye(n // block), 0.3 * np.eye(block) + 0.01 * (B + B.T))
    w, Z, _ = symeig_check(A, n)
    scale = np.abs(A).sum(axis=1).max()
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-11 * scale
    assert np.abs(A @ Z - Z * w[None, :]).max() <= 1e-10 * scale
    assert np.abs(Z.T @ Z - np.eye(n)).max() <= 1e-10
