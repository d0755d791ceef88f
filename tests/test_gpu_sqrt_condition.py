"""S^1/2 of ill-conditioned overlap matrices, below and above the size where one CTA
hands over to the product kernels: Tamm-Dancoff and iterative sTD-DFT solves (which
form it in different orders of products) accept or refuse a matrix alike, and what is
accepted has Loewdin orbitals orthonormal to about 1e-9, hence roots (linear in them,
with energies below 1 Eh) within 1e-8 Eh of the oracle's, whose S^1/2 comes from an
eigen-decomposition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with_spectrum(natoms, lowest):
    from stda_b200 import synth
    mol, ints = synth.random_molecule(natoms, seed=41 + natoms, with_ints=True)
    rng = np.random.default_rng(natoms)
    n = mol.nao
    U = synth.haar_orthogonal(n, rng)
    w = np.exp(rng.uniform(np.log(max(lowest, 1e-2)), 0.0, n))
    w[0], w[1] = lowest, 1.0
    S = (U * w) @ U.T
    S = 0.5 * (S + S.T)
    mol.C = ((U / np.sqrt(np.abs(w))) @ U.T) @ synth.haar_orthogonal(n, rng)
    return mol, (S,) + tuple(ints[1:])


def _solve(eng, kw):
    from stda_b200.engine import Std2gError
    try:
        return eng.solve(kw).omega
    except Std2gError as e:
        assert e.code == 5, e      # overlap matrix not positive definite
        return None


@pytest.mark.parametrize("natoms", [8, 40])
@pytest.mark.parametrize("lowest", [1e-2, 2e-3, 1e-3, 5e-4, 2e-4, 1e-4, 1e-5, 1e-7, -1e-3])
def test_one_verdict(natoms, lowest):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = _with_spectrum(natoms, lowest)
    base = dict(ax=0.5, e_thr_ev=9.0 if natoms < 20 else 6.0)
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    tda = _solve(eng, Keywords(nroots=3, solver=1, **base))
    rpa = _solve(eng, Keywords(nroots=3, solver=2, conv_tol=1e-7, rpa=True, **base))
    again = _solve(eng, Keywords(nroots=3, solver=1, **base))
    eng.close()
    assert (tda is None) == (rpa is None) == (again is None)
    if lowest >= 1e-2:
        assert tda is not None
    if lowest <= 1e-5:
        assert tda is None
    if tda is not None:
        ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**base))
        assert np.abs(tda - np.sort(np.linalg.eigvalsh(ref.A))[:3]).max() < 1e-8
