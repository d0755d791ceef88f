"""Eigenvectors of dense windows of up to 320 CSFs: orthonormal to the rounding of
sums of n products (2 sqrt(n) eps), as an eigen-decomposition gives them; and equal,
far apart molecules, whose roots are many-fold: roots against the oracle to 1e-10 Eh
(1e3 roundings of energies below 1 Eh), vectors orthonormal as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _orthonormal(X):
    n, k = X.shape
    assert np.abs(X.T @ X - np.eye(k)).max() <= 2 * np.sqrt(n) * 2.2e-16


@pytest.mark.parametrize("natoms,seed,nroots", [(6, 11, 0), (10, 15, 0), (10, 15, 20)])
def test_orthonormal_vectors(natoms, seed, nroots):
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=seed, with_ints=True)
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    sol = eng.solve(Keywords(ax=0.5, e_thr_ev=25.0, nroots=nroots, solver=1))
    X = eng.vectors()
    eng.close()
    assert X.shape[0] <= 320 and X.shape[1] == len(sol.omega)
    assert (np.diff(sol.omega) >= 0).all()
    _orthonormal(X)


def _far_copies(copies):
    """Copies of a bent H3 (3 AOs, one occupied orbital) 128 bohr apart, orbitals
    localised on each: triplet CSFs of different pairs of copies do not couple."""
    from stda_b200 import synth
    from stda_b200.integrals import ao_integrals
    from stda_b200.molden import Molecule
    one = np.array([[0.0, 0.0, 0.0], [1.5, 0.0, 0.25], [0.5, 1.75, -0.5]])
    xyz = np.vstack([one + [0.0, 0.0, 128.0 * q] for q in range(copies)])
    Z = np.ones(3 * copies, dtype=np.int32)
    mol = Molecule(Z=Z, xyz=xyz, shells=synth.basis_shells(Z), title="far copies of H3")
    ints = ao_integrals(mol)
    e, U = np.linalg.eigh(ints[0][:3, :3])
    C = ((U / np.sqrt(e)) @ U.T) @ synth.haar_orthogonal(3, np.random.default_rng(1))
    mol.C = np.zeros((mol.nao, mol.nao))
    for q in range(copies):
        for k in range(3):   # occupied orbitals of all copies first
            mol.C[3 * q:3 * q + 3, q if k == 0 else copies + 2 * q + k - 1] = C[:, k]
    mol.eps = np.concatenate([np.full(copies, -0.5), np.tile([0.1, 0.25], copies)])
    mol.occ = np.concatenate([np.full(copies, 2.0), np.zeros(2 * copies)])
    return mol, ints


@pytest.mark.parametrize("copies", [3, 4, 12])
def test_far_copies(copies):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = _far_copies(copies)
    kw = dict(ax=0.5, e_thr_ev=60.0, triplet=True)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    assert len(ref.omega) == 2 * copies ** 2
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    sol = eng.solve(Keywords(**kw))
    X = eng.vectors()
    eng.close()
    assert len(sol.omega) == len(ref.omega)
    assert np.abs(sol.omega - ref.omega).max() < 1e-10
    _orthonormal(X)
