"""CG products of the mixed dense response solve at the edges of their kernel: 3 to
30 columns, CSF counts on both sides of its row
blocks (1184, 2368).  alpha(w) of both forms is refined to FP64 residuals of 1e-10
relative, which enter alpha squared: 1e-8 relative leaves room for the systems'
condition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,ethr,nw", [(3, 20.0, 1), (7, 11.0, 2), (12, 9.0, 3), (18, 8.0, 4),
                                            (30, 7.0, 5), (36, 7.0, 8),
                                            (33, 7.0, 10), (36, 7.0, 2), (41, 7.0, 4), (50, 6.5, 1)])
def test_alpha(natoms, ethr, nw):
    from stda_b200 import synth
    from stda_b200.engine import FLAG_TENSOR_ALWAYS, Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    om = np.linspace(0.0, 0.05, nw)
    out = []
    for precision in (0, 1):
        eng = Engine(0, precision, flags=FLAG_TENSOR_ALWAYS if precision else 0)
        eng.load(boundary_inputs(mol, ints))
        out.append(eng.polarizability(Keywords(ax=0.5, e_thr_ev=ethr, rpa=True, solver=1), om)[0])
        eng.close()
    assert np.allclose(out[0], out[1], rtol=1e-8, atol=1e-8)
