"""A (hi, lo) batch advanced in calls of a few ticks, which keep no B2 sums, in longer ones, and in
one: the same bits, with and without a graph that fits the short calls."""
import numpy as np
import pytest

import dynamite_gb300 as D
from helpers import STATE_FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,order,Tmax", [(65, 9, 100.0), (128, 9, 1e3), (130, 5, 1e3)])
@pytest.mark.parametrize("ticks_per_launch", [1, 32])
@pytest.mark.parametrize("enqueue", [False, True])
def test_short_calls_equal_one(product_built, L, order, Tmax, ticks_per_launch, enqueue):
    grid = D.grid.generate(L, Tmax=Tmax, interp_order=order)
    qs = [D.Quench(p=3, p2=p2, lam=0.5, Gamma=0.5 + 0.05 * k) for k, p2 in enumerate((4, 4, 0))]
    a = D.Batch([grid], qs, ticks_per_launch=ticks_per_launch)
    b = D.Batch([grid], qs)
    calls = (1, 1, 2, 3, 4, 1, 7, 2, 40, 1, 3, 2, 1, 1, 1, 5, 3)
    for n in calls:
        if enqueue:
            a.enqueue(n)
        else:
            assert a.run(n) == n
    a.sync()
    b.run(sum(calls))
    for q in range(len(qs)):
        assert a.info(q) == b.info(q)
        sa, sb = a.download(q), b.download(q)
        for f in STATE_FIELDS:
            np.testing.assert_array_equal(getattr(sa, f), getattr(sb, f), err_msg=f)
    a.close()
    b.close()
