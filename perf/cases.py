"""The work that users of this framework have it do, as cases of fixed and drawn sizes.

Five kinds, each through the package's public entry points and the C ABI of
include/dyn.h:

* ``quench``: a driver that keeps the two-time history in its own device arrays
  (as RG-Evo does) takes RK steps of a fixed schedule with `Simulation.run`, has
  the new rows stored behind its own (dyn_state_rows_store_dev) and rolls the
  context back to where it was, so that a pass can be repeated;
* ``batch``: `Batch.run` advances many quenches with their own step controllers,
  then the newest row of every quench is read back;
* ``adjoint``: `adjoint_forward` and `adjoint_backward` with the gradients in the
  temperature, the coupling and the initial history, then the rollback;
* ``save``: what a save writes: the reference-order interpolation arrays, the
  right-hand side, r, the energy, and the energy of every row;
* ``resume``: a checkpoint loaded from device arrays and sparsified
  (dyn_state_upload_dev, `sparsifyNscale`, dyn_state_rows_store_dev).

The histories are smooth two-time functions with a plateau and an aging regime
on a time grid that grows as a quench's own does (steps from 1e-5 growing by 1 %,
then the step size of a delta_max = 1e-10 run, t**0.423 / 245); the seed draws the
plateau, the aging exponent, the temperature and the coupling.

Not returned: the embedded error estimate of a step.  It is a difference of two
nearly equal rows, of which only the order of magnitude is meant.
"""
import ctypes as C
import functools
import math
import random

import numpy as np
import torch

import dynamite_gb300 as D
from dynamite_gb300 import _lib

FIELDS = ("t1grid", "dtr", "QK", "QR", "dQK", "dQR", "rvec", "drvec")
WIDE = ("QK", "QR", "dQK", "dQR")
STAGES = {1: 7, 2: 10}


def stages_of(method):
    return STAGES[method] if method in STAGES else 4 * (method - 2)


def listed():
    return [
        # one RK54 step of the smallest grid in the tests: launches and latency
        dict(name="update_fp64_L64", kind="quench", precision="fp64", L=64, order=9, rows=300, steps=1, method=1,
             p=3, p2=4, log=False),
        # the plain FP64 quench at the benchmark's grid length
        dict(name="quench_fp64_L512", kind="quench", precision="fp64", L=512, order=9, rows=1500, steps=8, method=1,
             p=3, p2=4, log=False),
        # the largest grid of the benchmark's workloads, SSPRK(10,4), a long history
        dict(name="quench_fp64_L1024_ssprk", kind="quench", precision="fp64", L=1024, order=9, rows=6000, steps=3,
             method=2, p=3, p2=4, log=False),
        # the (hi, lo) form alone: an ordinary quench, and a long one on the largest grid
        dict(name="quench_df_L512", kind="quench", precision="mixed_df", L=512, order=9, rows=5000, steps=16,
             method=1, p=3, p2=4, log=False),
        dict(name="quench_df_L1024", kind="quench", precision="mixed_df", L=1024, order=9, rows=20000, steps=8,
             method=1, p=3, p2=4, log=False),
        # an odd grid length in the plain mixed form, which replays a schedule
        dict(name="quench_mixed_L257", kind="quench", precision="mixed", L=257, order=9, rows=1000, steps=16,
             method=1, p=3, p2=4, log=False),
        # the benchmark's batch: 64 quenches on one grid, two RK54 steps of each
        dict(name="batch64_df_L512", kind="batch", precision="mixed_df", lengths="512", quenches=64, rows=800,
             ticks=14),
        # a batch of mixed grid lengths, drawn as the 64-quench job draws them
        dict(name="batch64_df_mixed_lengths", kind="batch", precision="mixed_df", lengths="256,512,1024", quenches=64,
             rows=400, ticks=14),
        # a small batch in the plain mixed form
        dict(name="batch16_mixed_L256", kind="batch", precision="mixed", lengths="256", quenches=16, rows=600,
             ticks=28),
        # gradients through ten FP64 steps: forward and backward
        dict(name="adjoint_L512", kind="adjoint", L=512, order=9, rows=400, steps=10, p=3, p2=4),
        # the observables of a save
        dict(name="save_L512", kind="save", L=512, order=9, rows=2000, p=3, p2=4),
        # a checkpoint resumed and sparsified
        dict(name="resume_sparsify_L512", kind="resume", precision="fp64", L=512, order=9, rows=8000, variant="gpu"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("quench", "quench", "quench", "quench", "batch", "batch", "adjoint", "save", "resume"))
    p, p2 = rng.choice(((3, 4), (3, 4), (3, 0), (2, 4)))
    order = rng.choice((9, 9, 9, 5))
    if kind == "quench":
        prec = rng.choice(("fp64", "fp64", "mixed", "mixed_df", "mixed_df"))
        # log-space response: an option of the FP64 form, used where R stays positive
        return dict(kind=kind, precision=prec, L=_log_int(rng, 64, 800), order=order, rows=_log_int(rng, 100, 8000),
                    steps=rng.randint(1, 8), method=rng.choice((1, 1, 1, 2, 4)), p=p, p2=p2,
                    log=prec == "fp64" and rng.random() < 0.2)
    if kind == "batch":
        lengths = rng.choice((str(_log_int(rng, 64, 512)), "128,256", "256,512", str(2 * _log_int(rng, 32, 256))))
        return dict(kind=kind, precision=rng.choice(("mixed_df", "mixed_df", "mixed")), lengths=lengths,
                    quenches=rng.randint(2, 48), rows=_log_int(rng, 100, 500), ticks=rng.choice((7, 14, 21)))
    if kind == "adjoint":
        return dict(kind=kind, L=_log_int(rng, 64, 300), order=order, rows=_log_int(rng, 100, 600),
                    steps=rng.randint(2, 8), p=p, p2=p2)
    if kind == "save":
        return dict(kind=kind, L=_log_int(rng, 64, 700), order=order, rows=_log_int(rng, 100, 4000), p=p, p2=p2)
    return dict(kind=kind, precision=rng.choice(("fp64", "mixed_df")), L=_log_int(rng, 64, 512), order=order,
                rows=_log_int(rng, 500, 8000), variant=rng.choice(("gpu", "cpu", "cuda_host")))


# ---------------------------------------------------------------- inputs
def _grid(L, order):
    """The grid of a length, made for the times it can resolve (kept by the package, as a program
    keeps its Grid_data)."""
    Tmax = 10.0 if L < 80 else 100.0 if L < 112 else 1e3 if L < 176 else 1e5
    return D.grid.generate(L, Tmax=Tmax, interp_order=order)


@functools.lru_cache(maxsize=32)
def _times(n):
    """Row times and the step size of the next row: a quench's own growth."""
    t, dt = [0.0], 1e-5
    for _ in range(n - 1):
        t.append(t[-1] + dt)
        dt = min(1.01 * dt, max(1e-5, t[-1] ** 0.423 / 245.0))
    return np.array(t), dt


def _model(rng, p=3, p2=4, **kw):
    return D.Model(p=p, p2=p2, lam=rng.choice((0.3, 0.5, 0.7)), Gamma=rng.uniform(0.4, 1.0), **kw)


def _fprime(m, q):
    return m.lam * m.p * q ** (m.p - 1) + ((1 - m.lam) * m.p2 * q ** (m.p2 - 1) if m.p2 else 0.0)


def _fsecond(m, q):
    a = m.lam * m.p * (m.p - 1) * q ** (m.p - 2)
    return a + ((1 - m.lam) * m.p2 * (m.p2 - 1) * q ** (m.p2 - 2) if m.p2 else 0.0)


def _history(grid, n, m, rng, device, spare=0):
    """n rows C(t_k, theta t_k), R(t_k, theta t_k) with the staggered derivative rows, r and dr,
    in arrays with room for `spare` more rows."""
    q, a = rng.uniform(0.5, 0.8), rng.uniform(0.2, 0.6)
    t_np, _ = _times(n)
    f64 = dict(dtype=torch.float64, device=device)
    th = torch.as_tensor(grid.theta, **f64)[None, :]
    w = torch.as_tensor(grid.integ, **f64)[None, :]
    t = torch.as_tensor(t_np, **f64)
    L = grid.L
    out = {f: torch.zeros(((n + spare), L) if f in WIDE else (n + spare,), **f64) for f in FIELDS}

    def rows(tt):
        tt = tt[:, None]
        u = (1 - th) * tt
        age = ((1 + th * tt) / (1 + tt)) ** a
        dage = age * a * (th / (1 + th * tt) - 1 / (1 + tt))
        pl = q + (1 - q) / (1 + u)
        dpl = -(1 - q) * (1 - th) / (1 + u) ** 2
        fast = (1 + u) ** -1.5
        dfast = -1.5 * (1 - th) * (1 + u) ** -2.5
        return pl * age, age * fast, dpl * age + pl * dage, dage * fast + age * dfast

    for k0 in range(0, n, 4096):
        k1 = min(n, k0 + 4096)
        K, R, _, _ = rows(t[k0:k1])
        out["QK"][k0:k1], out["QR"][k0:k1] = K, R
        out["rvec"][k0:k1] = m.Gamma + t[k0:k1] * (w * (_fsecond(m, K) * R * K + _fprime(m, K) * R)).sum(1) \
            + _fprime(m, K[:, 0]) * K[:, 0] / m.T0
        prev = torch.cat([t[:1], t])[k0:k1]  # t_{k-1}
        dt = (t[k0:k1] - prev)[:, None]
        _, _, dK, dR = rows(prev)
        out["dQK"][k0:k1], out["dQR"][k0:k1] = dt * dK, dt * dR
    out["t1grid"][:n] = t
    if n > 2:
        out["dtr"][2:n] = (t[2:] - t[1:-1]) / (t[1:-1] - t[:-2])
        out["drvec"][2:n] = (t[2:] - t[1:-1]) * (out["rvec"][1:n - 1] - out["rvec"][:n - 2]) / (t[1:-1] - t[:-2])
    return out


def _dev(h, n):
    return _lib.StateDev(n, *[h[f].data_ptr() for f in FIELDS])


def _schedule(case):
    _, dt = _times(case["rows"])
    k = case["steps"]
    # a stabilised method takes larger steps than RK54
    dt = dt * (1.0 if case.get("method", 1) < 3 else 2.0)
    return np.full(k, dt), np.full(k, case.get("method", 1), dtype=np.int32)


def _sim(case, m, precision, spare):
    return D.Simulation(_grid(case["L"], case["order"]), m, precision=precision,
                        history_capacity=case["rows"] + spare + 2, log_response=bool(case.get("log", False)))


def _quench_list(case, rng):
    """(lengths, per quench: grid index, model): lengths cycle in a drawn order, the temperatures
    span [0.4, 1.0] and lambda cycles, as the 64-quench job sets them."""
    lengths = [int(x) for x in case["lengths"].split(",")]
    n = case["quenches"]
    shift = rng.random() * 0.05
    order = [k % len(lengths) for k in range(n)]
    random.Random(7).shuffle(order)
    models = [D.Model(p=3, p2=4, lam=(0.3, 0.5, 0.7)[b % 3], Gamma=0.4 + shift + 0.6 * b / max(n - 1, 1),
                      delta_max=1e-4) for b in range(n)]
    return lengths, order, models


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "batch":
        lengths, order, models = _quench_list(case, rng)
        grids = [_grid(L, 9) for L in lengths]
        rows = case["rows"]
        b = D.Batch(grids, [D.Quench(grid=g, p=m.p, p2=m.p2, lam=m.lam, Gamma=m.Gamma, delta_max=m.delta_max,
                                     capacity=rows + 3000) for g, m in zip(order, models)],
                    precision=case["precision"])
        dt = _times(rows)[1]
        for k, (g, m) in enumerate(zip(order, models)):
            h = _history(grids[g], rows, m, rng, "cuda")
            b.upload(k, D.State(*[h[f].reshape(-1).cpu().numpy() for f in FIELDS]), delta_t=dt, method=1)
        return dict(kind=kind, b=b, ticks=case["ticks"], order=order, lengths=lengths)
    m = _model(rng, case.get("p", 3), case.get("p2", 4))
    grid = _grid(case["L"], case["order"])
    spare = case.get("steps", 0)
    s = _sim(case, m, case.get("precision", "fp64"), spare)
    h = _history(grid, case["rows"], m, rng, "cuda", spare)
    torch.cuda.synchronize()
    st = dict(kind=kind, s=s, h=h, n=case["rows"], L=case["L"])
    if kind == "resume":
        st["out"] = {f: torch.zeros_like(v) for f, v in h.items()}
        st["variant"] = case["variant"]
        st["threshold"] = m.delta_max  # the driver's own
        torch.cuda.synchronize()
        return st
    dev = _dev(h, case["rows"])
    _lib.check(_lib.lib().dyn_state_upload_dev(s._h, C.byref(dev)), "dyn_state_upload_dev")
    if kind == "quench":
        st["sched"] = _schedule(case)
    elif kind == "adjoint":
        st["sched"] = _schedule(case)
        c = np.asarray(D.grid.lagrange_weights(grid.theta, 0.5))
        st["obj"] = dict(w_energy=1.0, w_r=0.5, c_K=c, c_R=0.25 * c)
    return st


# ------------------------------------------------------------------ passes
def run(st):
    return {"quench": _run_quench, "batch": _run_batch, "adjoint": _run_adjoint, "save": _run_save,
            "resume": _run_resume}[st["kind"]](st)


def _run_quench(st):
    s, n, h = st["s"], st["n"], st["h"]
    dts, methods = st["sched"]
    k = len(dts)
    tr = s.run(k, schedule=(dts, methods))
    dev = _dev(h, n + k)
    _lib.check(_lib.lib().dyn_state_rows_store_dev(s._h, n, k, C.byref(dev)), "dyn_state_rows_store_dev")
    s.rollbackState(k)
    out = {f: h[f][n:n + k] for f in ("t1grid", "QK", "QR", "dQK", "dQR", "rvec", "drvec")}
    out["energy"], out["qk0"] = tr["energy"], tr["qk0"]
    return out


def _run_batch(st):
    b, order, lengths = st["b"], st["order"], st["lengths"]
    b.run(st["ticks"])
    out = {}
    for g, L in enumerate(lengths):
        idx = [k for k, x in enumerate(order) if x == g]
        K, R = np.empty((len(idx), L)), np.empty((len(idx), L))
        for r, k in enumerate(idx):
            b.last_row(k, K[r], R[r])
        out[f"C{L}"], out[f"R{L}"] = K, R
    inf = b.infos()
    for f in ("t", "energy", "r", "qk0"):
        out[f] = np.array([i[f] for i in inf])
    out["n"] = np.array([i["n"] for i in inf])
    return out


def _run_adjoint(st):
    s, n = st["s"], st["n"]
    k = len(st["sched"][0])
    tr = s.adjoint_forward(k, schedule=st["sched"])
    grad, _ = s.adjoint_backward(**st["obj"])
    g = s.adjoint_history_grad(n)
    s.rollbackState(k)
    return dict(energy=tr["energy"], grad=grad, QK=g.QK, QR=g.QR, dQK=g.dQK, dQR=g.dQR, rvec=g.rvec, drvec=g.drvec)


def _run_save(st):
    s, h, n = st["s"], st["h"], st["n"]
    s.interpolate()
    K1, R1, r_int = s.interp(4), s.interp(5), s.interp(16)
    hK, hR = s.QKRstep()
    return dict(QKB1=K1, QRB1=R1, rint=r_int, hK=hK, hR=hR, r=s.rstep(), energy=s.energy(),
                energy_history=s.energy_history())


def _run_resume(st):
    s, h, o, n = st["s"], st["h"], st["out"], st["n"]
    dev = _dev(h, n)
    _lib.check(_lib.lib().dyn_state_upload_dev(s._h, C.byref(dev)), "dyn_state_upload_dev")
    k = s.sparsifyNscale(st["threshold"], st["variant"])
    dst = _dev(o, k)
    _lib.check(_lib.lib().dyn_state_rows_store_dev(s._h, 0, k, C.byref(dst)), "dyn_state_rows_store_dev")
    # the caller's arrays, whole: rows past the k kept ones are as they were (zero)
    return dict(o, kept=k)


# ------------------------------------------------------------------- work
def _stage_work(L, m, prec):
    """One right-hand side: the arithmetic of the gathers, Sigma and the convolutions per target
    (A1, A2: 8 m; B1: 20; B2: 16 m + 30; Sigma 48; products 24)."""
    return (24 * m + 122) * L * L


def _table_bytes(L, m, prec):
    w = {"fp64": 8, "mixed": 4, "mixed_df": 8}[prec]
    return 3 * L * L * (w * m + 4) + 8 * L * L


def work(case):
    kind = case["kind"]
    if kind == "batch":
        lengths, order, _ = _quench_list(case, random.Random(0))
        by = sum(_table_bytes(L, 10, case["precision"]) for L in lengths)
        by += sum(case["rows"] * lengths[g] * 32 for g in order)
        return {"bytes": by, "flops": case["ticks"] * sum(_stage_work(lengths[g], 10, "") for g in order)}
    L, m, n = case["L"], case["order"] + 1, case["rows"]
    hist = 32.0 * n * L
    if kind == "quench":
        k = case["steps"]
        return {"bytes": _table_bytes(L, m, case["precision"]) + hist + 32.0 * k * L,
                "flops": k * stages_of(case["method"]) * _stage_work(L, m, "")}
    if kind == "adjoint":
        # forward, the same again backwards, and the transposed stages at twice a stage's work
        return {"bytes": 2 * _table_bytes(L, m, "fp64") + 2 * hist,
                "flops": 4.0 * case["steps"] * 7 * _stage_work(L, m, "")}
    if kind == "save":
        return {"bytes": _table_bytes(L, m, "fp64") + 0.5 * hist + 16.0 * L * L, "flops": _stage_work(L, m, "")}
    return {"bytes": 2 * hist, "flops": 20.0 * n * L}


# ------------------------------------------------ the same in plain torch
RK54_A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
          [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
          [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
          [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
RK54_B = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0]
SSP_A = [[1 / 6 if (r <= 4 or c >= 5) else 1 / 15 for c in range(r)] for r in range(10)]
SSP_B = [1 / 10] * 10


class _Plain:
    """The right-hand side and the RK steps on 64-bit tensors; differentiable."""

    def __init__(self, grid, m, device):
        f64 = dict(dtype=torch.float64, device=device)
        L, d = grid.L, grid.depth
        self.L, self.m, self.device = L, m, device
        self.lam = torch.tensor(m.lam, **f64)
        self.Gamma = torch.tensor(m.Gamma, **f64)
        self.th = torch.as_tensor(grid.theta, **f64)
        self.w = torch.as_tensor(grid.integ, **f64)
        self.phi2 = torch.as_tensor(grid.phi2, **f64)
        tap = torch.arange(d, device=device)[None, :]
        self.ind = [torch.as_tensor(np.asarray(a, dtype=np.int64), device=device)[:, None] + tap
                    for a in (grid.indsA1, grid.indsA2, grid.indsB2)]
        self.wt = [torch.as_tensor(a, **f64).reshape(L * L, d) for a in (grid.wA1, grid.wA2, grid.wB2)]

    def f1(self, q):
        m = self.m
        return self.lam * m.p * q ** (m.p - 1) + ((1 - self.lam) * m.p2 * q ** (m.p2 - 1) if m.p2 else 0.0)

    def f2(self, q):
        m = self.m
        a = self.lam * m.p * (m.p - 1) * q ** (m.p - 2)
        return a + ((1 - self.lam) * m.p2 * (m.p2 - 1) * q ** (m.p2 - 2) if m.p2 else 0.0)

    def f3(self, q):
        m = self.m
        a = self.lam * m.p * (m.p - 1) * (m.p - 2) * (q ** (m.p - 3) if m.p >= 3 else 0.0)
        return a + ((1 - self.lam) * m.p2 * (m.p2 - 1) * (m.p2 - 2) * q ** (m.p2 - 3) if m.p2 >= 3 else 0.0)

    @staticmethod
    def _interval(t, pos):
        """Rows k, k+1 around each time (the last interval holds the last time) and the offset."""
        k = torch.clamp(torch.searchsorted(t, pos, right=True) - 1, 0, t.numel() - 2)
        return k, (pos - t[k]) / (t[k + 1] - t[k])

    def _hermite(self, t, ratio, k, x):
        """Weights on value k, value k+1, derivative row k+1 and derivative row k+2."""
        last = k + 2 >= t.numel()
        k2 = torch.where(last, k, k + 2)
        c0 = torch.where(last, 1 - x * x, 1 - 3 * x ** 2 + 2 * x ** 3)
        c1 = torch.where(last, x * x, 3 * x ** 2 - 2 * x ** 3)
        c2 = torch.where(last, x - x * x, x - 2 * x ** 2 + x ** 3)
        c3 = torch.where(last, torch.zeros_like(x), (x ** 3 - x ** 2) / torch.where(last, torch.ones_like(x), ratio[k2]))
        return k2, c0, c1, c2, c3

    def rhs(self, S):
        """S: (t, ratio, K, R, dK, dR, r, dr), rows first."""
        t, ratio, K, R, dK, dR, r, dr = S
        L, m = self.L, self.m
        T = t[-1]
        a1 = [(self.wt[0] * v[-1][self.ind[0]]).sum(1).reshape(L, L) for v in (K, R)]
        a2 = [(self.wt[1] * v[-1][self.ind[1]]).sum(1).reshape(L, L) for v in (K, R)]
        k, x = self._interval(t, self.th * T)
        k2, c0, c1, c2, c3 = self._hermite(t, ratio, k, x)
        mix = lambda v, dv: (c0[:, None] * v[k] + c1[:, None] * v[k + 1] + c2[:, None] * dv[k + 1] + c3[:, None] * dv[k2])
        b1 = [mix(K, dK), mix(R, dR)]
        rint = c0 * r[k] + c1 * r[k + 1] + c2 * dr[k + 1] + c3 * dr[k2]
        k, x = self._interval(t, self.phi2 * T)
        k2, c0, c1, c2, c3 = self._hermite(t, ratio, k, x)
        col = self.ind[2]

        def seg(v, row):
            return (self.wt[2] * v[row[:, None], col]).sum(1)
        b2 = [(c0 * seg(v, k) + c1 * seg(v, k + 1) + c2 * seg(dv, k + 1) + c3 * seg(dv, k2)).reshape(L, L)
              for v, dv in ((K, dK), (R, dR))]
        sk = [self.f1(g[0]) for g in (a1, a2, b1, b2)]
        sr = [self.f2(g[0]) * g[1] for g in (a1, a2, b1, b2)]
        cv = lambda f, g: (f * g) @ self.w
        tA, tR = T * self.th, T * (1 - self.th)
        q, qr, q0 = K[-1], R[-1], K[-1][0]
        rE, qb = rint[-1], b1[0][:, 0]
        d1 = qb * self.f1(q0) / m.T0 - q * rE + tR * cv(sr[1], b2[0]) + tA * (cv(sr[0], b1[0]) + cv(sk[0], b1[1]))
        d2 = self.f1(qb) * q0 / m.T0 + 2 * self.Gamma * qr + tR * cv(a2[1], sk[3]) \
            + tA * (cv(a1[1], sk[2]) + cv(a1[0], sr[2])) - q * rint
        hK = d1 + d2 * self.th
        hR = -qr * rE + tR * cv(sr[1], b2[1]) + (qr * rint - tR * cv(a2[1], sr[3])) * self.th
        return torch.stack([hK, hR])

    def rstep(self, t, K, R):
        return self.Gamma + (t * self.w * (self.f2(K) * R * K + self.f1(K) * R)).sum() + self.f1(K[0]) * K[0] / self.m.T0

    def drstep(self, t, K, R, dK, dR):
        s = self.f2(K) * R
        ds = self.f3(K) * R * dK + self.f2(K) * dR
        v = (self.w * (s * K + self.f1(K) * R)).sum() \
            + (t * self.w * (ds * K + self.f2(K) * dK * R + s * dK + self.f1(K) * dR)).sum()
        return v + (self.f2(K[0]) * dK[0] * K[0] + self.f1(K[0]) * dK[0]) / self.m.T0

    def energy(self, t, K, R):
        return -((t * self.w * self.f1(K) * R).sum() + self.f1(K[0]) / self.m.T0)

    def step(self, S, method, dt):
        A, B = (RK54_A, RK54_B) if method == 1 else (SSP_A, SSP_B)
        t, ratio, K, R, dK, dR, r, dr = S
        T0, prev = float(t[-1]), float(t[-1] - t[-2])
        g0 = torch.stack([K[-1], R[-1]])
        h, DR, cur = [], None, S
        cat = lambda v, row: torch.cat([v, row[None]])
        one = lambda v: torch.as_tensor(v, dtype=torch.float64, device=self.device)
        for s in range(len(B)):
            h.append(self.rhs(cur))
            if s == 0:
                DR = self.drstep(T0, g0[0], g0[1], h[0][0], h[0][1])
            row = A[s + 1] if s + 1 < len(B) else B
            g, gt = g0, T0
            for c, hh in zip(row, h):
                g, gt = g + (dt * c) * hh, gt + dt * c
            td = gt - T0
            cur = (cat(t, one(gt)), cat(ratio, one(td / prev)), cat(K, g[0]), cat(R, g[1]), cat(dK, td * h[0][0]),
                   cat(dR, td * h[0][1]), cat(r, self.rstep(gt, g[0], g[1])), cat(dr, td * DR))
        return cur


def _as_state(h, n):
    """The tensors in the order _Plain wants, rows first."""
    return tuple(h[f][:n] for f in FIELDS)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, rng, dev)
    if kind == "resume":
        return None
    grid = _grid(case["L"], case["order"])
    m = _model(rng, case.get("p", 3), case.get("p2", 4))
    n = case["rows"]
    h = _history(grid, n, m, rng, dev)
    if kind == "quench":
        if case["method"] > 2 or case["log"]:
            return None
        P = _Plain(grid, m, dev)
        S = _as_state(h, n)
        for dt in _schedule(case)[0]:
            S = P.step(S, case["method"], float(dt))
        names = dict(zip(FIELDS, S))
        out = {f: names[f][n:] for f in ("t1grid", "QK", "QR", "dQK", "dQR", "rvec", "drvec")}
        out["energy"] = torch.stack([P.energy(t, a, b) for t, a, b in zip(out["t1grid"], out["QK"], out["QR"])])
        out["qk0"] = out["QK"][:, 0]
        return out
    if kind == "save":
        P = _Plain(grid, m, dev)
        S = _as_state(h, n)
        t, ratio, K, R, dK, dR, r, dr = S
        k, x = P._interval(t, P.th * t[-1])
        k2, c0, c1, c2, c3 = P._hermite(t, ratio, k, x)
        mix = lambda v, dv: (c0[:, None] * v[k] + c1[:, None] * v[k + 1] + c2[:, None] * dv[k + 1] + c3[:, None] * dv[k2])
        hh = P.rhs(S)
        eh = torch.cat([-t[a:a + 4096] * ((P.f1(K[a:a + 4096]) * R[a:a + 4096]) @ P.w + P.f1(K[a:a + 4096, 0]) / m.T0)
                        for a in range(0, n, 4096)])
        return dict(QKB1=mix(K, dK).reshape(-1), QRB1=mix(R, dR).reshape(-1),
                    rint=c0 * r[k] + c1 * r[k + 1] + c2 * dr[k + 1] + c3 * dr[k2], hK=hh[0], hR=hh[1],
                    r=float(P.rstep(t[-1], K[-1], R[-1])), energy=float(P.energy(t[-1], K[-1], R[-1])),
                    energy_history=eh)
    if kind == "adjoint":
        return _exact_adjoint(case, grid, m, h, n, dev)
    return None


def _exact_adjoint(case, grid, m, h, n, dev):
    from torch.utils.checkpoint import checkpoint

    P = _Plain(grid, m, dev)
    lam, Gamma = P.lam.requires_grad_(True), P.Gamma.requires_grad_(True)
    S = list(_as_state(h, n))
    leaves = S[2:] = [v.clone().requires_grad_(True) for v in S[2:]]
    leaves = list(leaves)
    en = []
    for dt in _schedule(dict(case, method=1))[0]:
        S = checkpoint(lambda *s, dt=float(dt): P.step(s, 1, dt), *S, use_reentrant=False)
        en.append(P.energy(S[0][-1], S[2][-1], S[3][-1]))
    c = torch.as_tensor(np.asarray(D.grid.lagrange_weights(grid.theta, 0.5)), dtype=torch.float64, device=dev)
    J = en[-1] + 0.5 * S[6][-1] + c @ S[2][-1] + 0.25 * (c @ S[3][-1])
    g = torch.autograd.grad(J, [Gamma, lam] + leaves, allow_unused=True)
    g = [torch.zeros(()) if v is None else v for v in g]
    names = ("QK", "QR", "dQK", "dQR", "rvec", "drvec")
    out = dict(energy=torch.stack([e.detach() for e in en]), grad=torch.stack([g[0], g[1]]))
    out.update({f: v.reshape(-1) for f, v in zip(names, g[2:])})
    return out


def _exact_batch(case, rng, dev):
    lengths, order, models = _quench_list(case, rng)
    if case["ticks"] % 7:
        return None
    n, steps = case["rows"], case["ticks"] // 7
    dt = _times(n)[1]
    out = {f: [] for f in ("t", "energy", "r", "qk0")}
    for L in lengths:
        out[f"C{L}"], out[f"R{L}"] = [], []
    plains = {}
    for g, m in zip(order, models):
        grid = _grid(lengths[g], 9)
        h = _history(grid, n, m, rng, dev)
        P = plains.get(g)
        if P is None:
            P = plains[g] = _Plain(grid, m, dev)
        P.m = m
        P.lam = torch.tensor(m.lam, dtype=torch.float64, device=dev)
        P.Gamma = torch.tensor(m.Gamma, dtype=torch.float64, device=dev)
        S = _as_state(h, n)
        for _ in range(steps):
            S = P.step(S, 1, dt)
        t, K, R = S[0][-1], S[2][-1], S[3][-1]
        out[f"C{lengths[g]}"].append(K)
        out[f"R{lengths[g]}"].append(R)
        out["t"].append(t)
        out["energy"].append(P.energy(t, K, R))
        out["r"].append(S[6][-1])
        out["qk0"].append(K[0])
    out = {f: torch.stack(v) for f, v in out.items() if v}
    out["n"] = None
    return out
