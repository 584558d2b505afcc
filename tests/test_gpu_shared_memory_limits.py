"""The shared-memory limit of a kernel belongs to the process: a second, shorter batch or adjoint
context must leave the first one's launches as they were."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS

pytestmark = pytest.mark.gpu

M = dict(p=3, p2=4, lam=0.5, Gamma=0.6)


def test_two_live_batches(product_built):
    long, short = (D.grid.generate(L, Tmax=1e5, interp_order=1, cache=False) for L in (3060, 2700))
    first = D.Batch([long], [D.Quench(capacity=16, **M)])
    first.run(1)
    second = D.Batch([short], [D.Quench(capacity=16, **M)])
    second.run(8)
    first.run(7)
    s = D.Simulation(long, D.Model(**M), precision="mixed_df")
    s.init()
    s.run(1)
    a, b = first.download(0), s.download()
    assert a.t1grid.size >= 2
    for f in STATE_FIELDS:
        v = getattr(b, f)
        np.testing.assert_array_equal(getattr(a, f)[: v.size], v, err_msg=f)
    for x in (first, second, s):
        x.close()


def test_two_adjoint_contexts(product_built):
    sims = []
    for L, order in ((960, 1), (64, 9)):
        s = D.Simulation(D.grid.generate(L, Tmax=1e5 if L > 64 else 100.0, interp_order=order), D.Model(**M))
        s.init()
        s.adjoint_forward(2, schedule=(np.full(2, 1e-3), np.ones(2, dtype=np.int32)))
        sims.append(s)
    first = sims[0].adjoint_backward(w_energy=1.0)[0]
    sims[1].adjoint_backward(w_energy=1.0)
    again, stats = sims[0].adjoint_backward(w_energy=1.0)
    assert stats["recompute_mismatch"] == 0
    np.testing.assert_allclose(again, first, rtol=1e-12)  # the additions' order is free
    for s in sims:
        s.close()
