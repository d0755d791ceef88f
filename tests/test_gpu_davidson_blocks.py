"""Block sizes of the Davidson solver (wanted plus buffer roots) at the edges
of its small kernels' tiles: 32 / 33, 64 / 65 and 112 / 113 columns, against
the dense eigen-decomposition of the same matrix: with residuals below 1e-7,
eigenvalues agree to residual^2 / gap, well below 1e-9 Eh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(36, seed=11, with_ints=True)
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    kw = dict(ax=0.5, e_thr_ev=7.0)
    dense = eng.solve(Keywords(nroots=100, solver=1, **kw)).omega
    yield eng, kw, dense
    eng.close()


@pytest.mark.parametrize("nroots", [1, 26, 27, 51, 52, 90, 91])
def test_block_sizes(engine, nroots):
    from stda_b200.engine import Keywords
    eng, kw, dense = engine
    s = eng.solve(Keywords(nroots=nroots, solver=2, conv_tol=1e-7, **kw))
    assert np.abs(s.omega - dense[:nroots]).max() < 1e-9
    assert s.extras["resid"].max() < 1e-7
