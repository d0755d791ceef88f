"""FP64 PT selection at the edges of its blocks (32 primaries, 64 candidates,
groups of one primary, few rows), against the oracle: the same CSF list, the
lowered diagonal to 1e-11 Eh (sums of at most 1e4 terms below 1e-2 in another
order: 1e4 x 2e-16 x 1e-2 with room for the couplings' rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,ethr,triplet", [(2, 22.0, False), (4, 14.0, False), (7, 10.0, True),
                                                 (12, 9.0, False), (18, 8.0, False),
                                                 (18, 11.5, True), (26, 8.0, False)])
def test_selection(natoms, ethr, triplet):
    from oracle.stda_fp64 import Params, stda as oracle_stda
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=31 + natoms, with_ints=True)
    kw = dict(ax=0.5, e_thr_ev=ethr, triplet=triplet)
    ref = oracle_stda(mol.xyz4(), mol.C, mol.eps, mol.occ, mol.iaoat(), *ints, Params(**kw))
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    eng.solve(Keywords(nroots=1, solver=1, **kw))
    iconf, ed = eng.csf()
    eng.close()
    got = np.stack([iconf[:, 0] - 1, iconf[:, 1] - 1 - ref.no], axis=1)
    assert np.array_equal(got, ref.iconf)
    assert np.abs(ed - ref.ed).max() < 1e-11
