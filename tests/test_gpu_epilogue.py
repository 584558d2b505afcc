"""The stage epilogue at the edges of its 32-row blocks, and the next stage's positions, which
it and the gathers search outwards from the last interval instead of over the whole list."""
import numpy as np
import pytest

import dynamite_gb300 as D
import oracle as O
from helpers import STATE_FIELDS, rel_err

pytestmark = pytest.mark.gpu

TRAJ_TOL = 1e-10  # as the trajectories of the parity tests


@pytest.mark.parametrize("L", [24, 31, 32, 33, 95])
@pytest.mark.parametrize("method", [1, 2, 4])
def test_rows_at_block_edges(product_built, oracle_built, L, method):
    grid = D.grid.generate(L, Tmax=10.0, interp_order=5)
    s = D.Simulation(grid, D.Model(p=3, p2=4, lam=0.5, Gamma=0.6))
    s.init()
    steps = 6
    sched = (1e-4 * 1.3 ** np.arange(steps), np.full(steps, method, dtype=np.int32))
    tr = s.run(steps, schedule=sched)
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    p = O.Port(og, O.Model(p=3, p2=4, lam=0.5, Gamma=0.6), search_mode=1, threads=0)
    p.init_state()
    tp = p.run(steps, schedule=sched)
    a, b = s.download(), p.get_state()
    np.testing.assert_array_equal(a.t1grid, b.t1grid)
    for k in ("QK", "QR", "rvec"):
        assert rel_err(getattr(a, k), getattr(b, k)) < TRAJ_TOL, k
    assert rel_err(tr["energy"], tp["energy"]) < TRAJ_TOL
    s.close()


@pytest.mark.parametrize("L,Tmax", [(63, 10.0), (65, 100.0), (129, 1e3), (192, 1e5), (193, 1e5)])
def test_two_threads_a_target(product_built, oracle_built, L, Tmax):
    """The gathers' two threads a target: chunk edges and both sides of the length where one
    thread takes a target again."""
    grid = D.grid.generate(L, Tmax=Tmax)
    s = D.Simulation(grid, D.Model(p=3, p2=4, lam=0.5, Gamma=0.6))
    s.init()
    sched = (1e-4 * 1.3 ** np.arange(5), np.array([1, 1, 2, 1, 4], dtype=np.int32))
    tr = s.run(5, schedule=sched)
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    p = O.Port(og, O.Model(p=3, p2=4, lam=0.5, Gamma=0.6), search_mode=1, threads=0)
    p.init_state()
    tp = p.run(5, schedule=sched)
    a, b = s.download(), p.get_state()
    for k in ("QK", "QR", "rvec"):
        assert rel_err(getattr(a, k), getattr(b, k)) < TRAJ_TOL, k
    assert rel_err(tr["energy"], tp["energy"]) < TRAJ_TOL
    s.close()


# a short list, one whose intervals a step leaves by several at once, and an even one
@pytest.mark.parametrize("L,Tmax,n,factor", [(33, 10.0, 2, 1.0), (64, 100.0, 20, 1.5), (257, 1e5, 24, 1.0),
                                             (512, 1e5, 40, 1.2)])
@pytest.mark.parametrize("search", ["binary", "lower_bound"])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_df"])
def test_positions_equal_the_full_search(product_built, L, Tmax, n, factor, search, precision):
    """A state taken over by another context has its positions searched anew: the next step
    is the same, bit for bit."""
    grid = D.grid.generate(L, Tmax=Tmax)
    m = D.Model(p=3, p2=4, lam=0.5, Gamma=0.6)
    a = D.Simulation(grid, m, precision=precision, search=search)
    a.init()
    dt = 1e-4 * factor ** np.arange(n)
    a.run(n, schedule=(dt, np.ones(n, dtype=np.int32)))
    b = D.Simulation(grid, m, precision=precision, search=search)
    b.upload(a.download())
    for step in (dt[-1], 3 * dt[-1], dt[-1] / 7):
        a.update(1, float(step))
        b.update(1, float(step))
    sa, sb = a.download(), b.download()
    for f in STATE_FIELDS:
        np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
    a.close()
    b.close()
