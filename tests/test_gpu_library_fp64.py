"""STD2G_FLAG_LIBRARY_FP64: every FP64 product of a context goes to cuBLAS, and the
iterative solvers give the same roots on them.  Both stop at residuals below 1e-9, which bounds the distance of their
Tamm-Dancoff roots by 2e-9 Eh and of their sTD-DFT roots by 2e-7 (w^2 of an operator
below 10 Eh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engines(natoms, seed):
    from stda_b200 import synth
    from stda_b200.engine import FLAG_LIBRARY_FP64, Engine, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=seed, with_ints=True)
    b = boundary_inputs(mol, ints)
    for flags in (0, FLAG_LIBRARY_FP64):
        eng = Engine(0, 0, flags=flags)
        eng.load(b)
        yield eng
        eng.close()


@pytest.mark.parametrize("natoms,ethr,nroots,rpa", [(12, 9.0, 17, False), (30, 7.0, 25, False), (18, 8.0, 9, True)])
def test_iterative_roots(natoms, ethr, nroots, rpa):
    from stda_b200.engine import Keywords
    kw = Keywords(ax=0.5, e_thr_ev=ethr, nroots=nroots, solver=2, conv_tol=1e-9, rpa=rpa)
    own, lib = (eng.solve(kw) for eng in _engines(natoms, 61 + natoms))
    assert np.abs(own.omega - lib.omega).max() < (2e-7 if rpa else 2e-9)


@pytest.mark.parametrize("natoms,ethr,kw", [
    (7, 11.0, dict()), (18, 8.0, dict(nroots=9)), (18, 8.0, dict(solver=1)), (40, 7.0, dict(nroots=5)),
    (7, 11.0, dict(rpa=True)), (18, 8.0, dict(rpa=True, nroots=4)), (18, 8.0, dict(triplet=True, nroots=4))])
def test_no_product_on_the_own_kernels(natoms, ethr, kw):
    """... and the CSF space is the same: the PT sums differ by the order of their terms
    (at most 1e4 of them below 1e-2)."""
    from stda_b200.engine import Keywords
    k = Keywords(ax=0.5, e_thr_ev=ethr, **kw)
    seen = []
    for eng in _engines(natoms, 31 + natoms):
        eng.solve(k)
        seen.append((eng.gemm_launches()["own"], eng.gemm_stats()["calls"], eng.csf()))
    (own, _, (c0, e0)), (lib, calls, (c1, e1)) = seen
    assert own > 0 and lib == 0 and calls > 0
    assert np.array_equal(c0, c1) and np.abs(e0 - e1).max() < 1e-11


@pytest.mark.parametrize("solver", [1, 2])
def test_response_on_cublas(solver):
    """alpha(w), refined to residuals of 1e-10 relative in both forms."""
    from stda_b200.engine import Keywords
    out = []
    for eng in _engines(18, 49):
        out.append(eng.polarizability(Keywords(ax=0.5, e_thr_ev=8.0, rpa=True, solver=solver), np.array([0.0, 0.04]))[0])
        out.append(eng.gemm_launches()["own"])
    assert out[1] > 0 and out[3] == 0
    assert np.allclose(out[0], out[2], rtol=1e-8, atol=1e-8)
