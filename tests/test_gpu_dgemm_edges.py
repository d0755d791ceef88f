"""FP64 products at the edges of the kernel's tiles and K splits: partial last
K tiles, clamped rows and columns, sums split over many CTAs, and two members
a fixed distance apart.  Against numpy: |err| <= 4 eps (k + 8) |A| |B| summed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("m,n,k,b", [(1, 1, 1, 1), (63, 31, 15, 1), (65, 33, 17, 2), (64, 128, 64, 1),
                                     (25, 25, 3119, 1), (141, 40, 5945, 1), (300, 62, 20011, 1),
                                     (5001, 25, 13, 2), (17, 129, 128, 5)])
def test_edges(ta, tb, m, n, k, b):
    from stda_b200.engine import dgemm_check
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((b, k, m) if ta else (b, m, k))
    B = rng.standard_normal((b, n, k) if tb else (b, k, n))
    C = rng.standard_normal((b, m, n))
    out, _ = dgemm_check(A, B, C, ta, tb, alpha=-1.5, beta=0.5)
    a, bb = (A.transpose(0, 2, 1) if ta else A), (B.transpose(0, 2, 1) if tb else B)
    ref = -1.5 * np.matmul(a, bb) + 0.5 * C
    bound = 4 * 2.2e-16 * (k + 8) * (1.5 * np.matmul(np.abs(a), np.abs(bb)) + np.abs(C))
    assert np.all(np.abs(out - ref) <= bound)
