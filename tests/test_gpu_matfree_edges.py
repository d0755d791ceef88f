"""FP64 matrix-free products, whose atoms' products read and write the AO slots
of one atom inside AO-major arrays: iterative roots against the oracle's dense
diagonalisation, at sizes that put the occupied block and the slots times
vectors across the edges of the 64 x 32 tiles.  A residual norm of 1e-9 bounds the
error of a TDA root by 1e-9 Eh; sTD-DFT roots (w^2 is the eigenvalue, of an
operator of norm below 10 Eh, and w > 0.1 Eh) by 1e-7."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rpa", [False, True])
@pytest.mark.parametrize("natoms,ethr,nroots,ax", [(3, 20.0, 3, 0.5), (7, 11.0, 5, 0.2), (12, 9.0, 17, 0.5),
                                                   (18, 8.0, 9, 0.0), (30, 7.0, 25, 0.5)])
def test_roots(natoms, ethr, nroots, ax, rpa):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    kw = dict(ax=ax, e_thr_ev=ethr, rpa=rpa)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    n = min(nroots, len(ref.iconf), len(ref.omega))
    sol = eng.solve(Keywords(nroots=n, solver=2, conv_tol=1e-9, **kw))
    eng.close()
    assert np.abs(sol.omega[:n] - np.sort(ref.omega)[:n]).max() < (1e-7 if rpa else 1e-9)


@pytest.mark.parametrize("natoms,ethr", [(99, 6.5), (108, 6.5)])
def test_by_ao_form(natoms, ethr):
    """Several tiles of occupied (189 and 187) and virtual orbitals (109 and 116): roots
    and alpha(w) against the engine's explicit matrices.  Roots to the residual
    bound, alpha as the other matrix-free tests."""
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    kw = dict(ax=0.5, e_thr_ev=ethr)
    dense = eng.solve(Keywords(nroots=12, solver=1, **kw)).omega
    it = eng.solve(Keywords(nroots=12, solver=2, conv_tol=1e-9, **kw)).omega
    assert np.abs(it - dense[:12]).max() < 1.1e-9
    om = np.array([0.0, 0.05])
    a1, _ = eng.polarizability(Keywords(solver=1, rpa=True, **kw), om)
    a2, _ = eng.polarizability(Keywords(solver=2, rpa=True, **kw), om)
    eng.close()
    assert np.allclose(a1, a2, rtol=1e-8, atol=1e-8)
