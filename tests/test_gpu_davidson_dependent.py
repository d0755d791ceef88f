"""Iterative solver where the correction blocks do not fit into what is left of
the space: their Gram matrices have no Cholesky factor and the blocks go through
the eigen-decomposition that drops dependent directions.  Against the dense
eigenvalues of the oracle's matrices; residual norms of 1e-9 bound the errors as
1e-9 Eh (Tamm-Dancoff) and 1e-7 (sTD-DFT: w^2 of an operator below 10 Eh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,ethr,nroots,rpa", [(3, 20.0, 13, False), (7, 11.0, 70, False),
                                                    (12, 9.0, 150, False), (3, 20.0, 6, True),
                                                    (7, 11.0, 20, True)])
def test_dependent_blocks(natoms, ethr, nroots, rpa):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    kw = dict(ax=0.5, e_thr_ev=ethr, rpa=rpa)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    want = (np.sqrt(np.sort(np.linalg.eigvals(ref.Amb @ ref.Apb).real)) if rpa
            else np.linalg.eigvalsh(ref.A))[:nroots]
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    sol = eng.solve(Keywords(nroots=nroots, solver=2, conv_tol=1e-9, **kw))
    eng.close()
    assert np.abs(sol.omega - want).max() < (1e-7 if rpa else 1e-9)
