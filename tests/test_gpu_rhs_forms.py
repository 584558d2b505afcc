"""The right-hand side call, which keeps no B2 sums, against the first stage of a step from the
same state, which does; and a step after it against one without."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS, rel_err
from test_log_response import positive_history

pytestmark = pytest.mark.gpu

RHS_TOL = 1e-12  # as the right-hand sides of the parity tests


# both sides of the length where FP64 keeps them after all, chunk edges, one and two targets a
# thread, a generic depth, run-time exponents
@pytest.mark.parametrize("L,order,p2", [(64, 9, 4), (129, 9, 4), (192, 9, 4), (193, 9, 4), (257, 9, 0), (300, 5, 4),
                                        (512, 9, 5), (770, 9, 4)])
@pytest.mark.parametrize("precision,log_response", [("fp64", False), ("fp64", True), ("mixed", False), ("mixed_df", False)])
def test_rhs_equals_first_stage(product_built, L, order, p2, precision, log_response):
    grid = D.grid.generate(L, Tmax=100.0 if L < 100 else 1e3 if L < 200 else 1e5, interp_order=order)
    a, b = (D.Simulation(grid, D.Model(p=3, p2=p2, lam=0.5, Gamma=0.6), precision=precision, log_response=log_response)
            for _ in range(2))
    for s in (a, b):
        s.upload(positive_history(D.State, grid.theta, n=90, Tm=30.0))
    sched = (np.array([1e-3, 2e-3]), np.ones(2, dtype=np.int32))
    hK, hR = a.rhs()
    for s in (a, b):
        s.run(2, schedule=sched)
    sa, sb = a.download(), b.download()
    for f in STATE_FIELDS:
        np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
    row = slice(-2 * L, -L)  # of the first step
    tdiff = sa.t1grid[-2] - sa.t1grid[-3]
    if precision == "fp64":  # the call takes the reference's search, a stage the interval's stored inverse
        assert rel_err(sa.dQK[row], tdiff * hK) < RHS_TOL and rel_err(sa.dQR[row], tdiff * hR) < RHS_TOL
    else:
        np.testing.assert_array_equal(sa.dQK[row], tdiff * hK)
        np.testing.assert_array_equal(sa.dQR[row], tdiff * hR)
    for s in (a, b):
        s.close()
