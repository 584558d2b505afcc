"""The depth-10 mixed kernels at odd lengths, where a history row starts at either parity: a batch
against the same quenches alone, bit for bit, and the (hi, lo) form against FP64."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS, rel_err

pytestmark = pytest.mark.gpu

M = dict(p=3, p2=4, lam=0.5, Gamma=0.6)
TMAX = {65: 100.0, 66: 100.0, 129: 1e3, 257: 1e5}


@pytest.mark.parametrize("precision", ["mixed", "mixed_df"])
@pytest.mark.parametrize("lengths", [(65,), (257,), (65, 66, 129)])
def test_batch_equals_single_at_odd_lengths(product_built, precision, lengths):
    grids = [D.grid.generate(L, Tmax=TMAX[L]) for L in lengths]
    m = D.Model(**M)
    n = 12
    qs = [D.Quench(grid=g, p=m.p, p2=m.p2, lam=m.lam, T0=m.T0, Gamma=m.Gamma, delta_t_min=m.delta_t_min,
                   delta_max=m.delta_max, max_steps=n) for g in range(len(lengths)) for _ in range(2)]
    b = D.Batch(grids, qs, precision=precision)
    b.run(100_000)
    for q in range(len(qs)):
        s = D.Simulation(grids[qs[q].grid], m, precision=precision)
        s.init()
        s.run(n)
        sa, sb = b.download(q), s.download()
        for f in STATE_FIELDS:
            np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
        s.close()


@pytest.mark.parametrize("L", [65, 257])
def test_hi_lo_form_at_odd_lengths(product_built, L):
    grid = D.grid.generate(L, Tmax=TMAX[L])
    sched = (1e-4 * 1.3 ** np.arange(8), np.array([1, 1, 2, 1, 4, 1, 1, 2], dtype=np.int32))
    st = []
    for precision in ("fp64", "mixed_df"):
        s = D.Simulation(grid, D.Model(**M), precision=precision)
        s.init()
        s.run(8, schedule=sched)
        st.append(s.download())
        s.close()
    for f in ("QK", "QR", "rvec"):
        assert rel_err(getattr(st[1], f), getattr(st[0], f)) < 1e-9, f
