"""The status of the bounded tensor-core waits belongs to one call: a call that ended
with another error after a wait had run out leaves nothing that a later one reports."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_expired_wait_is_not_reported_twice():
    from stda_b200 import synth
    from stda_b200.engine import FLAG_TENSOR_ALWAYS, Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(12, seed=73, with_ints=True)
    base = dict(ax=0.5, e_thr_ev=9.0, solver=2)
    kw = Keywords(nroots=9, conv_tol=1e-7, **base)
    eng = Engine(0, 1, flags=FLAG_TENSOR_ALWAYS)
    eng.load(boundary_inputs(mol, ints))

    def both():
        return (eng.solve(kw).omega,
                eng.polarizability(Keywords(rpa=True, **base), np.array([0.0, 0.03]))[0])

    before = both()
    assert eng.lib.std2g_leave_expired_wait(eng.ctx) == 0
    after = both()
    eng.close()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
