"""A solve gives the same bits whatever was solved before on the same wavefunction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,precision", [(12, 0), (36, 0), (36, 1)])
def test_order_of_solves(natoms, precision):
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=71 + natoms, with_ints=True)
    b = boundary_inputs(mol, ints)
    base = dict(ax=0.5, e_thr_ev=7.5)
    tda = Keywords(nroots=12, conv_tol=1e-7, **base)
    rpa = Keywords(nroots=4, solver=2, conv_tol=1e-7, rpa=True, **base)

    def run(*what):
        eng = Engine(0, precision)
        eng.load(b)
        out = [eng.solve(k) for k in what]
        eng.close()
        return out

    def same(x, y):
        for f in ("omega", "fL", "fV", "RL", "RV", "alpha0"):
            assert np.array_equal(getattr(x, f), getattr(y, f)), f

    t1, r1, t2, r2 = run(tda, rpa, tda, rpa)
    r3, t3 = run(rpa, tda)
    same(t1, t2)
    same(t1, t3)
    same(r1, r2)
    same(r1, r3)
