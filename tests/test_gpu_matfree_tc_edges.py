"""Tensor-core matrix-free products at sizes whose orbital, AO-slot and vector
counts end inside the 128 x 128 x 64 tiles and their 8-element paddings: mixed-form
roots against the FP64 form's.  Both end on FP64 residuals below 1e-7, which bounds the
roots' errors by 1e-7 each; the velocity-corrected strengths (the exchange
products) agree to 1e-3 relative: vectors to 1e-7 over gaps above 1e-4 Eh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,ethr,nroots", [(3, 20.0, 3), (7, 11.0, 5), (12, 9.0, 17), (30, 7.0, 25),
                                                (41, 6.5, 9)])
def test_roots(natoms, ethr, nroots):
    from stda_b200 import synth
    from stda_b200.engine import FLAG_TENSOR_ALWAYS, Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    kw = Keywords(ax=0.5, e_thr_ev=ethr, nroots=nroots, solver=2, conv_tol=1e-7, velcorr=True)
    sols = []
    for precision in (0, 1):
        eng = Engine(0, precision, flags=FLAG_TENSOR_ALWAYS if precision else 0)
        eng.load(boundary_inputs(mol, ints))
        sols.append(eng.solve(kw))
        eng.close()
    a, b = sols
    assert np.abs(a.omega - b.omega).max() < 2e-7
    assert np.allclose(a.fV, b.fV, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("natoms,ethr", [(12, 9.0), (41, 6.5)])
def test_alpha(natoms, ethr):
    """The A+B, A-B products of alpha(w): both forms refine to FP64 residuals."""
    from stda_b200 import synth
    from stda_b200.engine import FLAG_TENSOR_ALWAYS, Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(natoms, seed=61 + natoms, with_ints=True)
    out = []
    for precision in (0, 1):
        eng = Engine(0, precision, flags=FLAG_TENSOR_ALWAYS if precision else 0)
        eng.load(boundary_inputs(mol, ints))
        out.append(eng.polarizability(Keywords(ax=0.5, e_thr_ev=ethr, rpa=True, solver=2),
                                      np.array([0.0, 0.03]))[0])
        eng.close()
    assert np.allclose(out[0], out[1], rtol=1e-7, atol=1e-7)
