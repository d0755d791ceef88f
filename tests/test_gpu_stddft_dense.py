"""Dense sTD-DFT on either side of the sizes where its square root and its
eigensolver change (96 CSFs, 320 CSFs): every root of the window, and a root
count, against the oracle's eigen-decompositions.  S^1/2 is good to
kappa(S) eps < 1e-11 and w^2 follows it linearly, so that an error of w grows as 1 / w."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,csfs", [(2, 8), (3, 25), (5, 61), (6, 105), (9, 209), (10, 216),
                                         (12, 321), (13, 395)])
@pytest.mark.parametrize("nroots", [0, 6])
def test_roots(natoms, csfs, nroots):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=5 + natoms, with_ints=True)
    kw = dict(ax=0.5, e_thr_ev=25.0, rpa=True)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    assert len(ref.omega) == csfs
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    # solver 1: the dense form at every size
    sol = eng.solve(Keywords(nroots=nroots, solver=1, **kw))
    eng.close()
    k = nroots or csfs
    assert len(sol.omega) == k
    tol = 1e-10 * np.maximum(1.0, 0.1 / ref.omega[:k])
    assert (np.abs(sol.omega - ref.omega[:k]) < tol).all()
