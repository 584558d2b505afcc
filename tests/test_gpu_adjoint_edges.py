"""The adjoint at the edges of its kernels: lengths around the warps that share a row, its
columns and the B2 packets' runs, a stencil depth without the run kernel, and exponents with
and without compile-time derivatives; against central differences as in test_gpu_adjoint."""
import numpy as np
import pytest

import dynamite_gb300 as D
from test_gpu_adjoint import _agree, _fd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,order,p,p2", [(24, 5, 3, 4), (31, 9, 3, 4), (32, 9, 3, 0), (33, 9, 2, 4), (65, 9, 3, 4)])
def test_adjoint_matches_fd_at_edges(product_built, L, order, p, p2):
    grid = D.grid.generate(L, Tmax=10.0, interp_order=order)
    m = D.Model(p=p, p2=p2, lam=0.5, Gamma=0.6)
    s = D.Simulation(grid, m)
    s.init()
    n = 8
    sched = (1e-4 * 1.5 ** np.arange(n), np.array([1, 1, 1, 2, 1, 2, 1, 1], dtype=np.int32))
    s.adjoint_forward(n, schedule=sched)
    cK = D.grid.lagrange_weights(grid.theta, 0.5)
    gE, stats = s.adjoint_backward(w_energy=1.0)
    assert stats["recompute_mismatch"] == 0
    adj = {"E": gE, "C": s.adjoint_backward(c_K=cK)[0], "r": s.adjoint_backward(w_r=1.0)[0]}
    fd = _fd(grid, m, sched, cK)
    for obj in ("E", "C", "r"):
        for k, name in enumerate(("Gamma", "lam")):
            a, f = adj[obj][k], fd[name][obj]
            assert _agree(a, f, fd["J"][obj], getattr(m, name)), (obj, name, a, f)
    s.close()
