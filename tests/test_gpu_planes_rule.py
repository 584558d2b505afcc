"""Where the plain mixed form keeps its B2 sums depends on the length, the history and the call:
the results do not, on both sides of each line and across one within a call."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS
from test_log_response import positive_history

pytestmark = pytest.mark.gpu


# up to 672 always; above, calls of four steps from 8 (L - 640) rows on, and odd lengths always
@pytest.mark.parametrize("L,rows,steps", [(672, 60, 2), (674, 60, 5), (674, 269, 7), (674, 300, 3), (674, 300, 4),
                                          (705, 60, 4)])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("use_graph", [True, False])
def test_run_equals_single_updates(product_built, L, rows, steps, method, use_graph):
    grid = D.grid.generate(L, Tmax=1e5)
    m = D.Model(p=3, p2=4, lam=0.5, Gamma=0.6)
    a, b = (D.Simulation(grid, m, precision="mixed", use_graph=use_graph) for _ in range(2))
    for s in (a, b):
        s.upload(positive_history(D.State, grid.theta, n=rows, Tm=30.0))
    dt = 1e-3 * 1.2 ** np.arange(steps)
    tr = a.run(steps, schedule=(dt, np.full(steps, method, dtype=np.int32)))
    for k in range(steps):
        r = b.update(method, float(dt[k]))
        assert (r.delta, r.energy, r.r) == (tr["delta"][k], tr["energy"][k], tr["r"][k])
    sa, sb = a.download(), b.download()
    for f in STATE_FIELDS:
        np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
    for s in (a, b):
        s.close()
