"""Statistics of the FP64 products: with timing on, each product that is counted is
also timed."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(nroots=20, conv_tol=1e-7), dict(solver=1), dict(rpa=True, solver=2, nroots=4)])
def test_every_counted_product_is_timed(kw):
    from stda_b200 import synth
    from stda_b200.engine import Engine, Keywords, boundary_inputs
    mol, ints = synth.random_molecule(18, seed=5, with_ints=True)
    k = Keywords(ax=0.5, e_thr_ev=8.0, **kw)
    eng = Engine(0, 0)
    eng.load(boundary_inputs(mol, ints))
    sol = eng.solve(k)           # S^1/2, once per load
    assert sol.nexpt > 0         # PT candidates: the (ij|ab) products are among the counted
    eng.set_gemm_timing(True)
    eng.solve(k)
    stats, seen = eng.gemm_stats(), eng.gemm_launches()
    eng.close()
    assert stats["calls"] > 0 and stats["ms"] > 0.0
    assert seen["timed"] == stats["calls"]
