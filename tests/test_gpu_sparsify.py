"""The sparsify indicator and the in-place compaction against the oracle, bit for bit: row
counts around a CTA's nodes, odd lengths, and values where the shared-divisor division has to
fall back to the general one (zero, tiny and huge derivatives, very short intervals)."""
import numpy as np
import pytest

import oracle as O
import dynamite_gb300 as D
from helpers import STATE_FIELDS

pytestmark = pytest.mark.gpu


def _state(cls, L, n, seed):
    r = np.random.default_rng(seed)
    t = np.concatenate([[0.0], np.cumsum(r.uniform(0.5, 1.5, n - 1) * 1e-3)])
    if n > 12:
        t[7:] -= t[7] - t[6] - 1e-160  # an interval too short for the fast division
    K = 1.0 + r.standard_normal((n, L)) * 1e-4
    R = 1.0 + r.standard_normal((n, L)) * 1e-4
    dK = r.standard_normal((n, L)) * 10.0 ** r.integers(-9, -3, (n, L))
    dR = r.standard_normal((n, L)) * 10.0 ** r.integers(-9, -3, (n, L))
    for a in (dK, dR):
        a[r.random((n, L)) < 0.05] = 0.0
        a[r.random((n, L)) < 0.05] *= 1e-290
    dK[0, 0] = 1e140
    dtr = np.zeros(n)
    with np.errstate(over="ignore", divide="ignore"):
        dtr[2:] = np.minimum((t[2:] - t[1:-1]) / (t[1:-1] - t[:-2]), 1e300)
    return cls(t, dtr, K.ravel(), R.ravel(), dK.ravel(), dR.ravel(), r.standard_normal(n), r.standard_normal(n) * 1e-4)


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("L,n", [(32, 3), (32, 4), (33, 18), (33, 19), (32, 35), (95, 67), (64, 300)])
def test_sparsify_equals_oracle(product_built, L, n, variant):
    grid = D.grid.generate(L, Tmax=10.0)
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    s = D.Simulation(grid, D.Model())
    p = O.Port(og, O.Model(), search_mode=1, threads=2)
    # twice on the same context: the workspace of the first pass serves a larger second one
    for k, rows in enumerate((max(3, n // 2), n)):
        st = _state(D.State, L, rows, 100 * n + k)
        s.upload(st)
        p.set_state(_state(O.State, L, rows, 100 * n + k))
        for thr in (7e-8 * L, 9e-8 * L):
            assert s.sparsifyNscale(thr, ["cpu", "cuda_host", "gpu"][variant]) == p.sparsify(thr, variant)[0]
            a, b = s.download(), p.get_state()
            for f in STATE_FIELDS:
                np.testing.assert_array_equal(getattr(a, f), getattr(b, f), err_msg=f)
    s.close()


@pytest.mark.parametrize("L", [32, 255, 257, 300])
def test_reference_order_sums_equal_oracle(product_built, L):
    """r, dr, the energy and QKRstep around the 256-column blocks of their ordered sums."""
    grid = D.grid.generate(L, Tmax=10.0 if L < 64 else 1e3)
    og = O.Grid(L, grid.theta, grid.phi1, grid.phi2, grid.integ, grid.indsA1, grid.wA1, grid.indsA2, grid.wA2,
                grid.indsB2, grid.wB2)
    m = dict(p=3, p2=4, lam=0.3, T0=1.7, Gamma=0.6)
    s = D.Simulation(grid, D.Model(**m))
    s.init()
    s.run(4, schedule=(np.full(4, 1e-3), np.ones(4, dtype=np.int32)))
    st = s.download()
    p = O.Port(og, O.Model(**m), search_mode=0, threads=2)
    p.set_state(O.State(*(getattr(st, f) for f in STATE_FIELDS)))
    p.interpolate()
    s.interpolate()
    hK, hR = s.QKRstep()
    np.testing.assert_array_equal(hK, p.qkstep())
    np.testing.assert_array_equal(hR, p.qrstep())
    assert s.rstep() == p.rstep()
    assert s.energy() == p.energy(st.t1grid[-1])
    t, qK, qR = st.t1grid[-1], st.QK[-L:], st.QR[-L:]
    assert s.drstep2(qK, qR, hK, hR, t) == p.drstep2(qK, qR, hK, hR, t)
