"""The engine's work as a user has it done: sizes, options and entry points.

Each case goes through the public Python API (``Engine``, ``Ensemble``,
``xpattern.direct_fourier``), whose arrays are host arrays as in the reference's
own binding; ``exact`` gives the same values from plain torch in 64 bits (on the
GPU when there is one): the pair field in a cancellation-free form, dense solves
by ``torch.linalg.solve`` and gradients by torch's autograd.

Kinds of case:
  step      one attempted implicit step (``Engine.attempt``): the unit every
            simulation consists of, from N=64 (the reference's fixture size) to
            N=4096; option sets: plain FP64, mixed form, tabulated field,
            distant-pair cutoff with GMRES
  run       accepted steps of a continued simulation (``restore``, ``advance``)
  sweeps    the stress sweep and the fused stress and Jacobian sweep alone
  solve     the linear-solver boundary: matrix in, factorise, two right-hand sides
  ensemble  a batch of realisations of uneven N: create, rounds, results
  adjoint   d strain / d (x0, tau0) over recorded steps
  xpattern  direct-Fourier pattern analysis of one configuration
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("2d4_b200")
ens_mod = importlib.import_module("2d4_b200.ensemble")
xp_mod = importlib.import_module("2d4_b200.xpattern")

# sizes over which each kind is drawn (even numbers, spread over their logarithm)
RANGES = {
    "step": (64, 4096),
    "mixed": (2048, 4096),
    "tabulated": (64, 2048),
    "cutoff": (512, 4096),
    "run": (64, 1536),
    "sweeps": (64, 4096),
    "solve": (64, 3072),
    "ensemble": (128, 2048),  # largest instance
    "adjoint": (64, 1024),
    "xpattern": (200, 4096),
}


def listed():
    return [
        # N=64, tight precision: the reference's own fixture size, where launches count
        dict(name="step64", kind="step", n=64, h=4e-6, tau=0.0, precision=1e-8),
        # a small odd size under cyclic load, dipole criterion off, other weight function
        dict(name="step250-cyclic", kind="step", n=250, h=1e-6, tau=0.0, precision=1e-6,
             cyclic=True, weight="p"),
        # the headline size: accepted steps under constant stress, continued from a saved state
        dict(name="run1024", kind="run", n=1024, h=2e-7, tau=0.05, precision=1e-5, steps=4),
        # the tabulated field at a size that is no multiple of a tile
        dict(name="step1000-table", kind="step", n=1000, h=5e-7, tau=0.05, precision=1e-5,
             table=1024),
        # the solver boundary as the UMFPACK calls use it
        dict(name="solve1500", kind="solve", n=1500),
        # stress and Jacobian sweeps alone, as an analysis script calls them
        dict(name="sweeps2000", kind="sweeps", n=2000, h=2e-7, tau=0.1),
        # N=4096 plain FP64: the largest dense system of the benchmark
        dict(name="step4096", kind="step", n=4096, h=1e-7, tau=0.1, precision=1e-5),
        # the same in the mixed form
        dict(name="step4096-mixed", kind="step", n=4096, h=1e-7, tau=0.1, precision=1e-5,
             mixed=True),
        # the same with the distant-pair cutoff (Heaviside, radius 0.1), solved by GMRES
        dict(name="step4096-cutoff", kind="step", n=4096, h=1e-7, tau=0.1, precision=1e-5,
             cutoff=0.1),
        # a batch of realisations of uneven N under a stress ramp
        dict(name="ensemble192", kind="ensemble", count=192, n=2048, rounds=2),
        # gradients of the strain at N=1024 over a few recorded steps, in two segments
        dict(name="adjoint1024", kind="adjoint", n=1024, steps=6, every=3, h=1e-7, tau=0.08),
        # pattern analysis at the tool's default resolution
        dict(name="xpattern4096", kind="xpattern", n=4096, res=1024),
    ]


def _size(rng, kind):
    lo, hi = RANGES[kind]
    return 2 * int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))


def draw(rng):
    kind = rng.choice(["step", "step", "mixed", "tabulated", "cutoff", "run", "sweeps", "solve",
                       "ensemble", "adjoint", "xpattern"])
    n = _size(rng, kind)
    h = math.exp(rng.uniform(math.log(2e-8), math.log(1e-6)))
    tau = rng.choice([0.0, 0.05, 0.1])
    if kind == "xpattern":
        return dict(kind=kind, n=n, res=rng.randrange(128, 1025))
    if kind == "ensemble":
        return dict(kind=kind, count=rng.randrange(8, 97), n=n, rounds=rng.choice([1, 2]))
    if kind == "solve":
        return dict(kind=kind, n=n)
    if kind == "sweeps":
        return dict(kind=kind, n=n, h=h, tau=tau)
    if kind == "adjoint":
        return dict(kind=kind, n=n, steps=rng.randrange(2, 6), every=rng.choice([2, 3, 20]), h=h,
                    tau=tau)
    if kind == "run":
        return dict(kind=kind, n=n, h=h, tau=tau, precision=1e-5, steps=rng.randrange(1, 5))
    case = dict(kind="step", n=n, h=h, tau=tau, precision=1e-5)
    if kind == "mixed":
        case["mixed"] = True
    elif kind == "tabulated":
        case["table"] = rng.choice([512, 1024])
    elif kind == "cutoff":
        case["cutoff"] = rng.choice([0.05, 0.1])
    else:
        case["weight"] = rng.choice(["c", "p", "m"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _positions(n, seed):
    """iid uniform positions, internal order: b = +1 first, y descending per sign."""
    r = np.random.default_rng(seed)
    x = r.uniform(-0.5, 0.5, n)
    y = r.uniform(-0.5, 0.5, n)
    y = np.concatenate([np.sort(y[:n // 2])[::-1], np.sort(y[n // 2:])[::-1]])
    return x, y


def _ensemble_configs(case, seed):
    """Sizes uniform over even values in [64, n], the same for every seed."""
    r = np.random.default_rng(case["count"])
    ns = 2 * r.integers(32, case["n"] // 2 + 1, size=case["count"])
    ns[0] = case["n"]
    return [_positions(int(n), 1000 * seed + 17 + k) for k, n in enumerate(ns)]


def _matrix(case, seed):
    """A Jacobian's shape: I plus a row-scaled symmetric coupling, as I + D J is."""
    n = case["n"]
    r = np.random.default_rng(seed)
    c = r.standard_normal((n, n)) / n
    c = (c + c.T) / 2
    d = 0.5 * (1 + r.uniform(0, 1, n))
    a = d[:, None] * c
    a[np.arange(n), np.arange(n)] = 1 + d * np.abs(c).sum(1)
    return np.asfortranarray(a), r.standard_normal((2, n))


def _steps(case):
    hs = case["h"] * 1.5 ** np.arange(case["steps"])
    return np.concatenate([[0.0], np.cumsum(hs)[:-1]]), hs


CYCLE = dict(rate=5.0, period=0.01)


def _cutoff_multiplier(case):
    return case["cutoff"] * math.sqrt(case["n"])


def _engine(case, x, y):
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    sd.precision = case.get("precision", 1e-5)
    sd.weight_function = case.get("weight", "c")
    if case.get("cyclic"):
        sd.external_stress = pkg.CyclicLoadProtocol(0.0, CYCLE["rate"], CYCLE["period"])
        sd.dipole_precision = 0.0
    else:
        sd.external_stress = pkg.FixedRateProtocol(case.get("tau", 0.0), 0.0)
    if case.get("mixed"):
        sd.precision_mode = pkg._lib.D4_PREC_MIXED
    if case.get("table"):
        sd.field = pkg._lib.D4_FIELD_TABULATED
        sd.table_size = case["table"]
    if case.get("cutoff"):
        sd.cutoff_multiplier = _cutoff_multiplier(case)
        sd.heaviside_cutoff = True
        sd.solver = pkg._lib.D4_SOLVER_GMRES
    return pkg.Engine(sd)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "ensemble":
        st["configs"] = _ensemble_configs(case, seed)
        sd = pkg.SimulationData()
        sd.external_stress = pkg.FixedRateProtocol(0.0, 1e-3)
        sd.time_limited, sd.time_limit = True, 200.0
        st["sd"] = sd
        return st
    st["x"], st["y"] = _positions(case["n"], seed)
    if kind == "xpattern":
        st["b"] = np.where(np.arange(case["n"]) < case["n"] // 2, 1.0, -1.0)
        return st
    st["engine"] = _engine(case, st["x"], st["y"])
    if kind == "solve":
        st["a"], st["g"] = _matrix(case, seed)
    if kind == "run":
        st["tol"] = st["engine"].tolerance()
    if kind == "adjoint":
        st["t0s"], st["hs"] = _steps(case)
    return st


def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "ensemble":
        ens = pkg.Ensemble(state["sd"], state["configs"])
        res = ens.run(case["rounds"])
        xs = [ens.positions(k)[0] for k in range(len(res))]
        ens.close()
        return {"x": np.concatenate(xs), "time": np.array([r.sim_time for r in res]),
                "step": np.array([r.step_size for r in res]),
                "accepted": np.array([r.successful_steps for r in res])}
    if kind == "xpattern":
        return xp_mod.direct_fourier(state["x"], state["y"], state["b"], case["res"])
    e, x, y = state["engine"], state["x"], state["y"]
    if kind == "step":
        r, xb, xh, x2 = e.attempt(0.0, case["h"])
        return {"big": xb, "half": xh, "two": x2, "ratio": r.ratio}
    if kind == "run":
        e.restore(x, y, 0.0, case["h"], state["tol"])
        r = e.advance(case["steps"])
        return {"x": e.positions()[0], "time": r.sim_time, "step": r.step_size}
    if kind == "sweeps":
        v, tol = e.speeds(x, y, 0.0)
        va, vb, _, d, _ = e.jacobian(x, y, case["h"], 0.0, case["h"], want_matrix=False)
        return {"v": v, "va": va, "vb": vb, "d": d, "tol": tol}
    if kind == "solve":
        e.set_matrix(state["a"])
        e.factor()
        return [e.solve(g)[0] for g in state["g"]]
    s, g, gt = e.adjoint(x, state["t0s"], state["hs"], case["every"])
    return {"strain": s, "grad": g, "grad_tau": gt}


# ---------------------------------------------------------------------------
# work: FLOP per unique pair of a stress sweep and of a fused stress and
# gradient sweep (each division, exp2 and cos one operation, as bench.py counts
# them), 2 N^3 / 3 per factorisation, 2 N^2 per solve
# ---------------------------------------------------------------------------
STRESS_PAIR, FUSED_PAIR = 136, 386


def _step_flops(n, dense=True):
    pairs = n * (n - 1) / 2
    f = pairs * (3 * STRESS_PAIR + 2 * FUSED_PAIR)
    return f + (3 * (2 * n ** 3 / 3) + 6 * 2 * n ** 2 if dense else 0)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        # instance sizes are uniform over [64, n]; their means of n, n^2, n^3
        lo, hi, c = 64.0, float(case["n"]), case["count"] * case["rounds"]
        w = max(hi - lo, 1.0)
        m1, m2, m3 = ((hi ** (k + 1) - lo ** (k + 1)) / ((k + 1) * w) for k in (1, 2, 3))
        pair = (3 * STRESS_PAIR + 2 * FUSED_PAIR) / 2 + 12
        return {"bytes": 24 * m1 * case["count"], "flops": c * (pair * m2 + 2 * m3)}
    n = case["n"]
    if kind == "xpattern":
        k = case["res"] // 2 + 1
        return {"bytes": 8 * (3 * n + 8 * k), "flops": 8.0 * n * k * k}
    if kind == "step":
        return {"bytes": 8 * 6 * n, "flops": _step_flops(n, not case.get("cutoff"))}
    if kind == "run":
        return {"bytes": 8 * 4 * n, "flops": case["steps"] * _step_flops(n)}
    if kind == "sweeps":
        return {"bytes": 8 * 9 * n, "flops": n * (n - 1) / 2 * (STRESS_PAIR + FUSED_PAIR)}
    if kind == "solve":
        return {"bytes": 8 * (n * n + 4 * n), "flops": 2 * n ** 3 / 3 + 4 * n ** 2}
    # adjoint: stages II and III forward (two factorisations, four solves, four
    # sweeps), four transposed solves and six derivative sweeps back
    pairs = n * (n - 1) / 2
    fwd = pairs * 2 * (STRESS_PAIR + FUSED_PAIR) + 2 * (2 * n ** 3 / 3) + 4 * 2 * n ** 2
    back = pairs * 6 * FUSED_PAIR + 4 * 2 * n ** 2
    return {"bytes": 8 * 2 * n, "flops": case["steps"] * (fwd + back)}


# ---------------------------------------------------------------------------
# exact: plain torch in 64 bits
# ---------------------------------------------------------------------------
PI = math.pi


def _t(a):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _image(u, s2, gradient, equal):
    """Image at distance u: stress 2 pi^2 u (ch c - 1) / (ch - c)^2 and the
    engine's x-derivative (sh taken as ch where `equal`), with ch - c and
    ch c - 1 formed from sinh^2 and sin^2, s2 = 2 sin^2(pi dy)."""
    a = 2 * torch.sinh(PI * u) ** 2
    q = a + s2
    n1 = a - s2 - a * s2
    w = n1 / (q * q)
    f = 2 * PI * PI * u * w
    if not gradient:
        return f, None
    sh = 1 + a if equal else torch.sinh(2 * PI * u)
    c = 1 - s2
    return f, 2 * PI * PI * (w + 2 * PI * u * (sh * c / (q * q) - 2 * w * sh / q))


def _field(dx, dy, gradient):
    s2 = 2 * torch.sin(PI * dy) ** 2
    f = torch.zeros_like(dx)
    g = torch.zeros_like(dx) if gradient else None
    for i in range(-3, 4):
        fi, gi = _image(dx + i, s2, gradient, abs(i) == 3)
        f = f + fi
        if gradient:
            g = g + gi
    neg = dx < 0
    sign = torch.where(neg, -torch.ones_like(dx), torch.ones_like(dx))
    dist = dx * sign  # |dx|
    f5, g5 = _image(dx - 5 * sign, s2, gradient, True)
    f4b, g4b = _image(dx + 4 * sign, s2, gradient, True)
    f4, g4 = _image(dx - 4 * sign, s2, gradient, True)
    f = f + f5 * dist + f4b * (1 - dist) + f4
    if gradient:
        g = g + g5 * dist + f5 * sign + g4b * (1 - dist) - f4b * sign + g4
    return f, g


def _wrap(v):
    return v - torch.floor(v + 0.5)


class _System:
    """One configuration's sweeps, stages and step control."""

    def __init__(self, case, x, y):
        n = len(x)
        self.n, self.case = n, case
        self.y = _t(y)
        self.b = torch.ones_like(self.y)
        self.b[n // 2:] = -1
        self.bb = self.b[:, None] * self.b[None, :]
        self.wfn = case.get("weight", "c")
        self.dipole = 0.0 if case.get("cyclic") else 0.05
        p = case.get("precision", 1e-5)
        self.min_prec = p * p / (self.dipole ** 2 if self.dipole else 1)
        self.radius2 = case["cutoff"] ** 2 if case.get("cutoff") else math.inf
        self.tol = torch.full_like(self.y, self.min_prec)

    def ext(self, t):
        if self.case.get("cyclic"):
            per, rate = CYCLE["period"], CYCLE["rate"]
            p = t - math.floor(t / per + 0.25) * per
            return rate * per / 2 - rate * p if p > per / 4 else rate * p
        return self.case.get("tau", 0.0) + self.case.get("rate", 0.0) * t

    def sweep(self, x, h=None, track=True):
        """Forces F (antisymmetric; row sums are the speeds without external
        stress) and, with h, the raw Jacobian h b b xy_diff_x (symmetric)."""
        n = self.n
        dx = _wrap(x[:, None] - x[None, :])
        dy = _wrap(self.y[:, None] - self.y[None, :])
        upper = torch.ones(n, n, dtype=torch.bool, device=x.device).triu(1)
        dx = torch.where(upper, dx, torch.full_like(dx, 0.25))
        dy = torch.where(upper, dy, torch.full_like(dy, 0.25))
        r2 = dx * dx + dy * dy
        if track and self.dipole:
            d = torch.where(upper, r2, torch.full_like(r2, math.inf)).detach()
            near = torch.minimum(d.min(0).values, d.min(1).values)
            self.tol = torch.minimum(self.tol, near)
        f, g = _field(dx, dy, h is not None)
        zero = torch.zeros_like(f)
        f = torch.where(upper, f * self.bb, zero)
        force = f - f.T
        if h is None:
            return force.sum(1), None
        g = torch.where(upper & (r2 < self.radius2), h * g * self.bb, zero)
        return force.sum(1), g + g.T

    def weight(self, s):
        p = torch.clamp(s, min=0)
        if self.wfn == "c":
            return (p / (p + 1)) ** 2
        if self.wfn == "p":
            return p / (p + 1)
        q = torch.where(p > 0, p, torch.ones_like(p))
        return torch.where(p > 0, 1 / (1 + 1.5 / (q + 0.412073 * q * q)), torch.zeros_like(p))

    def matrix(self, raw):
        sub = -raw.sum(1)
        d = self.weight(sub)
        sc = (1 + d) / 2
        return sc[:, None] * raw + torch.diag(1 + sub * sc), d

    def stage(self, base, y_end, v_init, hv, raw, ta, tb, speeds_end):
        """Two Newton iterations of one implicit stage of size hv from base."""
        a, d = self.matrix(raw)
        lu = torch.linalg.lu_factor(a)

        def solve(g):
            return torch.linalg.lu_solve(*lu, g[:, None])[:, 0]

        x1 = base - solve(-hv * ((1 + d) * y_end + (1 - d) * v_init) / 2)
        s1 = speeds_end(x1)
        return x1 - solve(x1 - base - hv * ((1 + d) * s1 + (1 - d) * v_init) / 2)

    def halves(self, x, t0, h, first=None):
        """Stages II and III."""
        b, e0, e1, eh = self.b, self.ext(t0), self.ext(t0 + h), self.ext(t0 + h / 2)
        v, raw = first if first is not None else self.sweep(x, h)
        xh = self.stage(x, v + eh * b, v + e0 * b, h / 2, raw / 2, t0, t0 + h / 2,
                        lambda z: self.sweep(z)[0] + eh * b)
        v2, raw2 = self.sweep(xh, h / 2)
        x2 = self.stage(xh, v2 + e1 * b, v2 + eh * b, h / 2, raw2, t0 + h / 2, t0 + h,
                        lambda z: self.sweep(z)[0] + e1 * b)
        return xh, x2

    def attempt(self, x, t0, h):
        b, e0, e1 = self.b, self.ext(t0), self.ext(t0 + h)
        first = self.sweep(x, h)
        v, raw = first
        xb = self.stage(x, v + e1 * b, v + e0 * b, h, raw, t0, t0 + h,
                        lambda z: self.sweep(z)[0] + e1 * b)
        xh, x2 = self.halves(x, t0, h, first)
        err = (xb - x2) ** 2
        ratio = float((err / self.tol).max()) / self.dipole ** 2 if self.dipole else float(
            (err / self.min_prec).max())
        return xb, xh, x2, ratio

    def next_step(self, x, t, h):
        """One attempt with its step control: positions, time, step, accepted."""
        _, _, x2, ratio = self.attempt(x, t, h)
        self.tol = torch.full_like(self.y, self.min_prec)
        hn = 0.9 * h * min(2.0, ratio ** (-1 / 6))
        return (_wrap(x2), t + h, hn, 1) if ratio < 1 else (x, t, hn, 0)


def _np(t):
    return t.detach().cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        xs, ts, hs, oks = [], [], [], []
        for x, y in _ensemble_configs(case, seed):
            s = _System(dict(rate=1e-3), x, y)
            z, t, h, ok = _t(x), 0.0, 1e-6, 0
            for _ in range(case["rounds"]):
                z, t, h, acc = s.next_step(z, t, h)
                ok += acc
            xs.append(_np(z))
            ts.append(t)
            hs.append(h)
            oks.append(ok)
        return {"x": np.concatenate(xs), "time": np.array(ts), "step": np.array(hs),
                "accepted": np.array(oks)}
    if kind == "solve":
        a, g = _matrix(case, seed)
        x = torch.linalg.solve(_t(a), _t(g).T).T
        return [_np(x[0]), _np(x[1])]
    x, y = _positions(case["n"], seed)
    if kind == "xpattern":
        k = torch.arange(case["res"] // 2 + 1, dtype=torch.float64, device=_t(x).device)

        def waves(v):
            ph = torch.remainder(_t(v)[:, None] * k[None, :], 1.0)
            return torch.exp(-2j * PI * ph)

        ex, ey, half = waves(x), waves(y), case["n"] // 2
        fp, fn = ey[:half].T @ ex[:half], ey[half:].T @ ex[half:]
        return np.stack([_np((f.abs() ** 2).sum(0)) for f in (fp + fn, fp - fn, fp, fn)])
    s = _System(case, x, y)
    if kind == "step":
        xb, xh, x2, ratio = s.attempt(_t(x), 0.0, case["h"])
        return {"big": _np(xb), "half": _np(xh), "two": _np(x2), "ratio": ratio}
    if kind == "run":
        z, t, h, ok = _t(x), 0.0, case["h"], 0
        while ok < case["steps"]:
            z, t, h, acc = s.next_step(z, t, h)
            ok += acc
        return {"x": _np(z), "time": t, "step": h}
    if kind == "sweeps":
        v, raw = s.sweep(_t(x), case["h"])
        tol = s.tol
        _, d = s.matrix(raw)
        v = _np(v + s.ext(0.0) * s.b)
        return {"v": v, "va": v, "vb": _np(_t(v)), "d": _np(d), "tol": _np(tol)}
    # adjoint: the replay step by step, gradients through torch's autograd
    t0s, hs = _steps(case)
    tau = torch.tensor(case["tau"], dtype=torch.float64, device=s.y.device)

    def step(z, tv, t0, h):
        s.ext = lambda t: tv
        _, x2 = s.halves(z, t0, h)
        return x2

    s.dipole = 0.0
    zs, strain = [_t(x)], 0.0
    with torch.no_grad():
        for t0, h in zip(t0s, hs):
            x2 = step(zs[-1], tau, t0, h)
            strain += float((s.b * (x2 - zs[-1])).sum())
            zs.append(_wrap(x2))
    lam, gt = torch.zeros_like(zs[0]), 0.0
    for k in range(len(hs) - 1, -1, -1):
        z = zs[k].clone().requires_grad_(True)
        tv = tau.clone().requires_grad_(True)
        out = (step(z, tv, t0s[k], hs[k]) * (lam + s.b)).sum() - (s.b * z).sum()
        lam, dt = torch.autograd.grad(out, (z, tv))
        gt += float(dt)
    return {"strain": strain, "grad": _np(lam), "grad_tau": gt}
