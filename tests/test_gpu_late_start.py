"""Histories on which a position is not simply inside its interval: starting after t = 0, so that
early positions lie before the first time, or with a time that repeats.  FP64 steps against the
oracle and against the right-hand side of the same state, whose search is the reference's."""
import numpy as np
import pytest

import dynamite_gb300 as D
import oracle as O
from helpers import rel_err
from test_log_response import T_ROWS, time_history_state

pytestmark = pytest.mark.gpu

TRAJ_TOL = 1e-10  # as the trajectories of the parity tests
RHS_TOL = 1e-12  # as the right-hand sides of the parity tests
M = dict(p=3, p2=4, lam=0.5, Gamma=0.6)
DTS = np.array([0.05, 0.02])
# both sides of the length where two threads share a target, one and two targets a thread
LENGTHS = [(65, False), (65, True), (257, False), (770, False)]


def _history(cls, L, late):
    st = time_history_state(cls, L)
    st.t1grid = T_ROWS + 0.75 if late else np.where(np.arange(T_ROWS.size) == 1, 0.0, T_ROWS)
    st.dtr = np.concatenate([[0.0, 0.0], np.full(T_ROWS.size - 2, 1.25)])
    return st


def _grid(L):
    return D.grid.generate(L, Tmax=100.0 if L < 100 else 1e5)


@pytest.mark.parametrize("L,log_response", LENGTHS)
@pytest.mark.parametrize("method", [1, 2])
def test_late_start_equals_oracle(product_built, oracle_built, L, log_response, method):
    grid = _grid(L)
    s = D.Simulation(grid, D.Model(**M), log_response=log_response)
    s.upload(_history(D.State, L, True))
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    p = O.Port(og, O.Model(**M), search_mode=1, threads=0, log_response=log_response)
    p.set_state(_history(O.State, L, True))
    p.interpolate()
    for dt in DTS:  # the second step goes on from the first one's sums
        p.update(method, float(dt))
    s.run(2, schedule=(DTS, np.full(2, method, dtype=np.int32)))
    a, b = s.download(), p.get_state()
    assert np.isfinite(b.QK).all() and np.isfinite(b.QR).all()
    for k in ("QK", "QR", "dQK", "dQR", "rvec"):
        assert rel_err(getattr(a, k), getattr(b, k)) < TRAJ_TOL, k
    s.close()


# (a repeated first time has no finite position under the reference's binary search)
@pytest.mark.parametrize("L,log_response", LENGTHS)
@pytest.mark.parametrize("late,search", [(True, "binary"), (True, "lower_bound"), (False, "lower_bound")])
def test_first_stage_equals_rhs(product_built, L, log_response, late, search):
    """A step's derivative row is its length times the right-hand side at its start."""
    sims = [D.Simulation(_grid(L), D.Model(**M), search=search, log_response=log_response) for _ in range(2)]
    for s in sims:
        s.upload(_history(D.State, L, late))
    two = np.full(2, 2, dtype=np.int32)
    hK, hR = sims[0].rhs()
    sims[0].run(1, schedule=(DTS[:1], two[:1]))
    st = sims[0].download()
    tdiff = st.t1grid[-1] - st.t1grid[-2]
    assert rel_err(st.dQK[-L:], tdiff * hK) < RHS_TOL and rel_err(st.dQR[-L:], tdiff * hR) < RHS_TOL
    hK, hR = sims[0].rhs()
    sims[1].run(2, schedule=(DTS, two))
    st = sims[1].download()
    tdiff = st.t1grid[-1] - st.t1grid[-2]
    assert rel_err(st.dQK[-L:], tdiff * hK) < RHS_TOL and rel_err(st.dQR[-L:], tdiff * hR) < RHS_TOL
    for s in sims:
        s.close()
