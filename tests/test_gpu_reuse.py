"""What the stages of one call keep from each other -- the B2 stencil sums of targets whose
rows did not change, and after an RK54 step its last right-hand side as the next step's
first -- changes no bit: `run` over several steps against the same steps taken by one
`update` call each, which starts from the history alone."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS

pytestmark = pytest.mark.gpu


def _growing(n, dt, factor):
    return dt * factor ** np.arange(n)


# lengths around the tile shapes: below one warp, odd, one tile and one more, several chunks
# per row; steps that stay within an interval (factor 1) and that outgrow the ones before
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_df"])
@pytest.mark.parametrize("L,Tmax,order", [(24, 10.0, 5), (33, 10.0, 9), (64, 100.0, 9), (65, 100.0, 9), (128, 1e3, 9),
                                          (130, 1e3, 5), (257, 1e5, 9), (514, 1e5, 9), (770, 1e5, 9)])
@pytest.mark.parametrize("methods", [(1,) * 14, (2,) * 6, (1, 1, 2, 2, 4, 4, 1, 1, 1, 2, 1, 1)])
def test_run_equals_single_updates(product_built, precision, L, Tmax, order, methods):
    grid = D.grid.generate(L, Tmax=Tmax, interp_order=order)
    m = D.Model(p=3, p2=4, lam=0.5, Gamma=0.6)
    sched = (_growing(len(methods), 1e-4, 1.3), np.array(methods, dtype=np.int32))
    a = D.Simulation(grid, m, precision=precision)
    b = D.Simulation(grid, m, precision=precision)
    a.init()
    b.init()
    tr = a.run(len(methods), schedule=sched)
    for k, (dt, meth) in enumerate(zip(*sched)):
        r = b.update(int(meth), float(dt))
        assert (r.delta, r.energy, r.r) == (tr["delta"][k], tr["energy"][k], tr["r"][k])
    # and again from the later state, after a rollback that leaves stale sums behind
    for s in (a, b):
        s.rollbackState(3)
    again = (np.full(5, sched[0][-1] / 3), np.ones(5, dtype=np.int32))
    a.run(5, schedule=again)
    for dt, meth in zip(*again):
        b.update(int(meth), float(dt))
    sa, sb = a.download(), b.download()
    for f in STATE_FIELDS:
        np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
    a.close()
    b.close()


@pytest.mark.parametrize("log_response,p2", [(False, 0), (True, 4)])
def test_run_equals_single_updates_options(product_built, log_response, p2):
    """The same with the log-space response, other exponents, and the controller's own steps."""
    grid = D.grid.generate(96, Tmax=100.0)
    m = D.Model(p=3, p2=p2, lam=0.5, Gamma=0.6, delta_max=1e-8)
    a = D.Simulation(grid, m, log_response=log_response)
    b = D.Simulation(grid, m, log_response=log_response, use_graph=False)
    a.init()
    b.init()
    tr = a.run(60)
    for dt, meth in zip(tr["dt"], tr["method"]):
        b.update(int(meth), float(dt))
    sa, sb = a.download(), b.download()
    for f in STATE_FIELDS:
        np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
