"""S^1/2 around the size where one CTA hands over to the product kernels (96
AOs) and at the edges of its 8 x 8 tiles: all roots of the window against the
oracle, which takes S^1/2 from an eigen-decomposition.  S^1/2 is good to about
kappa(S) eps < 1e-11, and the roots follow it linearly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms", [1, 2, 3, 4, 6, 9, 24, 25, 26, 27, 28])
def test_roots(natoms):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=5 + natoms, with_ints=True)
    kw = dict(ax=0.5, e_thr_ev=25.0 if natoms < 5 else 8.0)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    sol = eng.solve(Keywords(**kw))
    eng.close()
    assert len(sol.omega) == len(ref.omega)
    assert np.abs(sol.omega - ref.omega).max() < 1e-10
