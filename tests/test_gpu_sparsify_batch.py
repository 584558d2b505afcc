"""Sparsify passes of a batch over histories of very different lengths through one workspace: the
same rows as alone, and no more staging than its 64 MB."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS
from test_log_response import positive_history

pytestmark = pytest.mark.gpu

M = dict(p=3, p2=4, lam=0.5, Gamma=0.6, delta_max=1e-12)


def test_workspace_over_mixed_lengths(product_built):
    torch = pytest.importorskip("torch")
    grids = [D.grid.generate(L, Tmax=1e5 if L > 64 else 10.0, interp_order=3) for L in (1000, 32)]
    rows = (3200, 8192)  # about 2,190 of the long rows stay: two chunks of staging
    states = [positive_history(D.State, g.theta, n=n, t_hi=5.0, Tm=30.0) for g, n in zip(grids, rows)]
    b = D.Batch(grids, [D.Quench(grid=k, max_steps=2, capacity=n + 8, **M) for k, n in enumerate(rows)],
                sparsify_every=1, precision="mixed")
    for k, st in enumerate(states):
        b.upload(k, st, 1e-3, 1)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    b.run(1000)
    used = free - torch.cuda.mem_get_info()[0]
    for k, st in enumerate(states):
        s = D.Simulation(grids[k], D.Model(**M), precision="mixed")
        s.upload(st)
        s.set_controller(1e-3, 1)
        s.run(2, sparsify_every=1)
        sa, sb = b.download(k), s.download()
        assert sa.t1grid.size < rows[k]
        for f in STATE_FIELDS:
            np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
        s.close()
    b.close()
    # 64 MB of rows, the lists of 8,200 rows, and what the driver takes to load the kernels
    assert used < 96 << 20, used
