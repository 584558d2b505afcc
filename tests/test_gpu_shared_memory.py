"""Row lengths around the 48 KB of shared memory that a launch may use unasked: the staged row (16
bytes a column, 24 in log space) and the kernel's own arrays (up to 2 KB) count together."""
import numpy as np
import pytest

import dynamite_gb300 as D
import oracle as O
from helpers import rel_err

pytestmark = pytest.mark.gpu

TRAJ_TOL = 1e-10  # as the trajectories of the parity tests


# below the boundary, in the window where only the kernel's own arrays cross it, above it
@pytest.mark.parametrize("L,log_response", [(2944, False), (2975, False), (3050, False), (3072, False),
                                            (1960, True), (2000, True), (2048, True)])
def test_fp64_step_at_long_rows(product_built, oracle_built, L, log_response):
    grid = D.grid.generate(L, Tmax=1e5, interp_order=1, cache=False)
    s = D.Simulation(grid, D.Model(p=3, p2=4, lam=0.5, Gamma=0.6), log_response=log_response)
    s.init()
    sched = (np.array([1e-3]), np.array([1], dtype=np.int32))
    tr = s.run(1, schedule=sched)
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    p = O.Port(og, O.Model(p=3, p2=4, lam=0.5, Gamma=0.6), search_mode=0, threads=0, log_response=log_response)
    p.init_state()
    tp = p.run(1, schedule=sched)
    a, b = s.download(), p.get_state()
    for k in ("QK", "QR", "rvec"):
        assert rel_err(getattr(a, k), getattr(b, k)) < TRAJ_TOL, k
    assert rel_err(tr["energy"], tp["energy"]) < TRAJ_TOL
    s.close()
