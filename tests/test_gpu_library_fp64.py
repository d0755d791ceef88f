"""STD2G_FLAG_LIBRARY_FP64: the iterative solvers give the same roots on cuBLAS's
products.  Both stop at residuals below 1e-9, which bounds the distance of their
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
