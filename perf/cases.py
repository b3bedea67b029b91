"""The work that programs have this package do, as cases that can be timed and compared.

Every case integrates seeded synthetic planetary systems (nbg.workloads) through the package's public calls:

  steps       intr(s, n; grad)               a few steps of one system
  time        intr(s, t; grad)               one system to a time, with the fractional last step
  transits    intr(s, tt; grad)              one system with transit times and their derivatives
  parameters  intr(s, tp; grad)              the same with sky velocity and impact parameter
  cartesian   intr(s, out)                   one system, the state and Jacobian of every step
  device      Batch.run_device               equal systems kept on the GPU between calls
  host        Batch.run                      systems of mixed size from host arrays
  serve       Server.submit / result         independent requests of mixed size
  init        init_nbody_batch               initial conditions from orbital elements

listed() stands for the range of each; draw() spreads sizes over the same ranges.

Outputs are what the calls compute: state, Jacobian, transit arrays and counts.  The compensation terms of the
Kahan sums (xerror, verror, jac_error) are not among them: they are the rounding residues of x, v and jac_step,
below those arrays' last digit, and stand for no number of their own.

exact() restates the integration in plain numpy: AHL21 steps on dual numbers (value and derivatives with respect
to every initial coordinate and mass, and to the step), the Kepler drift by Stumpff series, transit times as roots
of the sky projection over a partial step.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package, whose folder's name is no Python identifier, registered as nbg."""
    if "nbg" not in sys.modules:
        folder = os.path.join(ROOT, "nbodygradient.jl_gb300")
        spec = importlib.util.spec_from_file_location("nbg", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules["nbg"] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules["nbg"])
    return sys.modules["nbg"]


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: a few steps of a two-body system inside a caller's own loop
        {"name": "steps_2body", "kind": "steps", "n": 2, "steps": 16, "grad": True, "kick": False},
        # an orbit without derivatives, e.g. a stability check
        {"name": "time_5body_nograd", "kind": "time", "n": 5, "steps": 301, "grad": False, "kick": False},
        # one likelihood evaluation: 1000 days of a two-planet system, 2000 steps
        {"name": "transits_3body", "kind": "transits", "n": 3, "steps": 2000, "grad": True, "kick": False},
        # the same for a compact seven-planet system, a stretch of its data
        {"name": "transits_8body", "kind": "transits", "n": 8, "steps": 400, "grad": True, "kick": False},
        # planet pairs advanced by kicks, star-planet pairs by Kepler drifts
        {"name": "kick_4body", "kind": "transits", "n": 4, "steps": 250, "grad": True, "kick": True},
        # photodynamics: sky velocity and impact parameter beside each transit time
        {"name": "parameters_6body", "kind": "parameters", "n": 6, "steps": 203, "grad": True, "kick": False},
        # a trajectory with the Jacobian of every step
        {"name": "cartesian_3body", "kind": "cartesian", "n": 3, "steps": 500, "grad": True, "kick": False},
        # the benchmark batch: 4096 three-body systems over 2000 steps
        {"name": "device_3body_4096", "kind": "device", "n": 3, "systems": 4096, "steps": 2000, "grad": True},
        # the compact systems as a batch, a stretch of their 1600 days
        {"name": "device_8body_1024", "kind": "device", "n": 8, "systems": 1024, "steps": 200, "grad": True},
        # a sample of mixed systems from host arrays: 2 to 10 bodies, uneven lengths, no two groups alike
        {"name": "host_uneven_203", "kind": "host", "n": 10, "systems": 203, "steps": 80, "grad": True},
        # independent requests, half of them with derivatives
        {"name": "serve_24", "kind": "serve", "n": 10, "systems": 24, "steps": 96, "grad": True},
        # the initial conditions of a batch
        {"name": "init_5body_4096", "kind": "init", "n": 5, "systems": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "time", "transits", "transits", "parameters", "cartesian", "device", "device",
                       "host", "serve", "init"])
    n = rng.randint(2, 10)
    if kind in ("steps", "time", "transits", "parameters", "cartesian"):
        most = {"steps": 256, "cartesian": 500}.get(kind, 2000)
        steps = _log_int(rng, 16, max(32, min(most, int(12000 / (n * n)))))
        grad = True if kind == "cartesian" else rng.random() < 0.7
        kick = kind != "cartesian" and n >= 3 and rng.random() < 0.2
        return {"kind": kind, "n": n, "steps": steps, "grad": grad, "kick": kick}
    if kind == "device":
        n = rng.choice([2, 3, 3, 4, 5, 6, 8, 10])
        systems = _log_int(rng, 16, 4096 if n <= 4 else 1024)
        # at most about half the work of the 4096-system batch
        most = 0.5 * 4096 * 2000 * 27 / (systems * n ** 3)
        return {"kind": kind, "n": n, "systems": systems,
                "steps": _log_int(rng, 32, max(48, min(2000, most, 12000 / (n * n)))), "grad": rng.random() < 0.75}
    if kind == "host":
        return {"kind": kind, "n": rng.randint(4, 10), "systems": _log_int(rng, 8, 256),
                "steps": _log_int(rng, 24, 96), "grad": rng.random() < 0.75}
    if kind == "serve":
        return {"kind": kind, "n": rng.randint(4, 10), "systems": _log_int(rng, 4, 32),
                "steps": _log_int(rng, 24, 96), "grad": True}
    return {"kind": kind, "n": n, "systems": _log_int(rng, 16, 4096)}


# ---------------------------------------------------------------- inputs

def _elements(case, seed):
    """(elements, h, steps) of each system of the case, from the workloads' own draws."""
    W = _package().workloads
    kind, n = case["kind"], case["n"]
    count = case.get("systems", 1)
    if kind in ("host", "serve"):
        # body counts and lengths are the case's own, whatever the seed: 2..n in turn, a quarter to all of the steps
        lengths = np.random.default_rng(count).integers(max(16, case["steps"] // 4), case["steps"] + 1, count)
        own = {b: W.batch_uneven(count, seed=seed, nmin=b, nmax=b) for b in range(2, n + 1)}
        return [(own[b][0][q], own[b][1][q], int(k))
                for q, (b, k) in enumerate(zip((2 + q % (n - 1) for q in range(count)), lengths))]
    if n == 3 and kind != "init":
        els, h, _ = W.batch_3body(count, seed)
        hs = [h] * count
    elif n == 8 and kind != "init":
        els, h, _ = W.batch_8body(count, seed)
        hs = [h] * count
    else:
        els, hs, _ = W.batch_uneven(count, seed=seed, nmin=n, nmax=n)
    return [(el, h, case.get("steps", 0)) for el, h in zip(els, hs)]


def _span(case, h, steps):
    """What the call integrates to: a whole number of steps, and for intr(s, time) a fraction more."""
    return h * (steps + 0.37) if case["kind"] == "time" else h * steps


def _pair(case, n):
    """pair[i, j] = 1 (a kick) for the planet pairs of a kick case; all Kepler otherwise."""
    p = np.zeros((n, n), dtype=np.uint8, order="F")
    if case.get("kick"):
        p[1:, 1:] = 1
    return p


def _states(case, seed):
    """One State per system (host-side initial conditions), with its h, steps and ElementsIC."""
    nbg = _package()
    out = []
    for el, h, steps in _elements(case, seed):
        ic = nbg.workloads.ic_of(el)
        s = nbg.State(ic)
        s.pair[...] = _pair(case, s.n)
        out.append((s, ic, h, steps))
    return out


def _ntt(steps):
    """Transit slots of a system of so many steps of a twentieth of its shortest period, whatever the seed."""
    return steps // 20 + 6


STATE_IN = ("t", "x", "v", "m", "xerror", "verror", "jac_step", "jac_error", "dqdt", "pair", "jac_init")
UPDATED = ("t", "x", "v", "xerror", "verror", "jac_step", "jac_error", "dqdt")
TRANSITS = ("tt", "dtdq0", "dtdelements", "count")


def _filled_batch(case, seed):
    """A Batch with its inputs filled in; its initial conditions come from init_nbody_batch, as for any batch."""
    nbg = _package()
    systems = _elements(case, seed)
    ics = [nbg.workloads.ic_of(el) for el, _, _ in systems]
    spans = [h * k for _, h, k in systems]
    n = [ic.nbody for ic in ics]
    b = nbg.Batch(n, 0, [h for _, h, _ in systems], spans, [_ntt(k) for _, _, k in systems],
                  bool(case["grad"]))
    for q, (x, v, jac) in enumerate(nbg.init_nbody_batch(ics)):
        b.view("x", q)[:] = x.ravel(order="F")
        b.view("v", q)[:] = v.ravel(order="F")
        b.view("m", q)[:] = ics[q].m
        b.view("jac_init", q)[:] = jac.ravel(order="F")
        b.view("jac_step", q)[:: 7 * n[q] + 1] = 1.0
    return b


def prepare(case, seed):
    nbg = _package()
    kind = case["kind"]
    if kind == "init":
        return {"case": case, "ics": [nbg.workloads.ic_of(el) for el, _, _ in _elements(case, seed)]}
    if kind == "device":
        b = _filled_batch(case, seed)
        held = {k: torch.from_numpy(b.arrays[k]).cuda() for k in STATE_IN}
        work = {k: t.clone() if k in UPDATED else t for k, t in held.items()}
        for k in TRANSITS:
            work[k] = torch.zeros(b.arrays[k].shape, device="cuda", dtype=torch.int64 if k == "count" else torch.float64)
        return {"case": case, "batch": b, "held": held, "work": work}
    if kind == "host":
        b = _filled_batch(case, seed)
        return {"case": case, "batch": b, "held": {k: b.arrays[k].copy() for k in UPDATED}}
    if kind == "serve":
        # a small service: 32 slots a group
        return {"case": case, "requests": _states(case, seed),
                "server": nbg.Server(slots_per_group=32, hbm_budget_bytes=8 << 30)}
    s, ic, h, steps = _states(case, seed)[0]
    span = _span(case, h, steps)
    return {"case": case, "s": s, "ic": ic, "span": span, "steps": steps, "intr": nbg.Integrator(nbg.ahl21, h, 0.0, span)}


# ---------------------------------------------------------------- one pass

def _state_out(s, grad):
    out = {"t": s.t, "x": s.x, "v": s.v}
    if grad:
        out.update(jac_step=s.jac_step, dqdt=s.dqdt)
    return out


def run(state):
    nbg = _package()
    case = state["case"]
    kind = case["kind"]
    grad = case.get("grad", True)
    if kind == "init":
        got = nbg.init_nbody_batch(state["ics"])
        return {"x": np.stack([g[0] for g in got]), "v": np.stack([g[1] for g in got]),
                "jac_init": np.stack([g[2] for g in got])}
    if kind == "device":
        b, work = state["batch"], state["work"]
        for k in UPDATED:
            work[k].copy_(state["held"][k])
        for k in TRANSITS:
            work[k].zero_()
        torch.cuda.current_stream().synchronize()  # the call runs on the library's own streams
        b.run_device(work)
        keep = ("t", "x", "v", "tt", "count") + (("jac_step", "dqdt", "dtdq0", "dtdelements") if grad else ())
        return {**{k: work[k] for k in keep}, "status": b.status}
    if kind == "host":
        b = state["batch"]
        for k in UPDATED:
            b.arrays[k][...] = state["held"][k]
        b.arrays["count"][...] = 0
        b.run()
        keep = ("t", "x", "v", "tt", "count") + (("jac_step", "dqdt", "dtdq0", "dtdelements") if grad else ())
        return {**{k: b.arrays[k].copy() for k in keep}, "status": b.status.copy()}
    if kind == "serve":
        srv, asked = state["server"], []
        for q, (s0, ic, h, steps) in enumerate(state["requests"]):
            s, tt = s0.copy(), nbg.TransitTiming(h * steps, ic, ntt=_ntt(steps))
            asked.append((srv.submit(s, tt, nbg.Integrator(nbg.ahl21, h, 0.0, h * steps), q % 2 == 0), s, tt))
        for rid, s, tt in asked:
            srv.result(rid, s, tt)
        flat = lambda get, which: np.concatenate([get(a).ravel(order="F") for a in which])  # noqa: E731
        return {"x": flat(lambda a: a[1].x, asked), "v": flat(lambda a: a[1].v, asked),
                "tt": flat(lambda a: a[2].tt, asked), "count": flat(lambda a: a[2].count, asked),
                "jac_step": flat(lambda a: a[1].jac_step, asked[::2]), "dqdt": flat(lambda a: a[1].dqdt, asked[::2]),
                "dtdq0": flat(lambda a: a[2].dtdq0, asked[::2]),
                "dtdelements": flat(lambda a: a[2].dtdelements, asked[::2])}
    s, intr = state["s"].copy(), state["intr"]
    if kind == "steps":
        intr(s, state["steps"], grad=grad)
        return _state_out(s, grad)
    if kind == "time":
        intr(s, float(state["span"]), grad=grad)
        return _state_out(s, grad)
    if kind == "cartesian":
        out = nbg.CartesianOutput(s.n, state["steps"])
        intr(s, out)
        return {**_state_out(s, True), "out_t": out.t, "out_x": out.x, "out_v": out.v, "out_jac": out.jac_step}
    if kind == "transits":
        tt = nbg.TransitTiming(state["span"], state["ic"], ntt=_ntt(state["steps"]))
        intr(s, tt, grad=grad)
        out = {**_state_out(s, grad), "tt": tt.tt, "count": tt.count}
        if grad:
            out.update(dtdq0=tt.dtdq0, dtdelements=tt.dtdelements)
        return out
    tp = nbg.TransitParameters(state["span"], state["ic"], ntt=_ntt(state["steps"]))
    intr(s, tp, grad=grad)
    out = {**_state_out(s, grad), "ttbv": tp.ttbv, "count": tp.count}
    if grad:
        out.update(dtbvdq0=tp.dtbvdq0, dtbvdelements=tp.dtbvdelements)
    return out


def work(case):
    """Inputs read and outputs written once; the flops of the Kepler solves (about 250 each), and with derivatives
    of the Jacobian updates: per column of jac_step the pair differences, the 6x6 products and their sums, the
    corrector's velocity-by-position block and the two drifts."""
    kind = case["kind"]
    count = case.get("systems", 1)
    if kind == "init":
        n = case["n"]
        return {"bytes": 8.0 * count * (7 * n + 6 * n + 49 * n * n), "flops": count * (1000.0 * n + 2 * 7.0 * 49 * n ** 3)}
    mixed = kind in ("host", "serve")
    total = {"bytes": 0.0, "flops": 0.0}
    for n in (range(2, case["n"] + 1) if mixed else [case["n"]]):
        share = count / (case["n"] - 1) if mixed else count
        steps = 0.625 * case["steps"] if mixed else case["steps"]
        grad = 0.5 if kind == "serve" else float(case["grad"])
        pairs, ntt, rows = n * (n - 1) / 2, steps / 20 + 3, 3 if kind == "parameters" else 1
        outs = 0 if kind in ("steps", "time", "cartesian") else rows * n * ntt * (1 + grad * 14 * n)
        if kind == "cartesian":
            outs = steps * (6 * n + 49 * n * n)
        total["bytes"] += 8 * share * (2 * 6 * n + n + grad * (3 * 49 * n * n + 7 * n) + outs)
        column = 2 * pairs * 96 + 18 * n * n + 12 * n
        total["flops"] += share * steps * (2 * pairs * 250 + grad * 7 * n * column)
    return total


# ---------------------------------------------------------------- the same in plain numpy
#
# A dual number is an array whose first axis holds the value and then its derivatives.

GNEWT = 39.4845 / (365.242 * 365.242)
_C2 = [1.0 / math.factorial(2 + 2 * k) * (-1) ** k for k in range(15)]
_C3 = [1.0 / math.factorial(3 + 2 * k) * (-1) ** k for k in range(15)]


def _mul(a, b):
    r = a * b[:1]
    r += a[:1] * b
    r[0] *= 0.5
    return r


def _func(a, value, slope):
    r = a * slope
    r[0] = value
    return r


def _inv(a):
    v = 1.0 / a[0]
    return _func(a, v, -v * v)


def _sqrt(a):
    v = np.sqrt(a[0])
    return _func(a, v, 0.5 / v)


def _dot(a, b):
    return _mul(a, b).sum(axis=-2, keepdims=True)


def _horner(c, z):
    p, d = np.full_like(z, c[-1]), np.zeros_like(z)
    for q in c[-2::-1]:
        d = d * z + p
        p = p * z + q
    return p, d


def _plain_horner(c, z):
    p = np.full_like(z, c[-1])
    for q in c[-2::-1]:
        p = p * z + q
    return p


def _kepler(x, v, k, h, drift_first):
    """Change of a relative orbit over a Kepler drift of h and a free drift of -h, in this order or the other."""
    xd = x - _mul(h, v) if drift_first else x
    r0 = _sqrt(_dot(xd, xd))
    r0inv = _inv(r0)
    eta = _dot(xd, v)
    beta = 2 * _mul(k, r0inv) - _dot(v, v)
    zeta = k - _mul(r0, beta)
    s = h[0] * r0inv[0]
    for _ in range(12):  # r0 s + eta G2 + zeta G3 = h, values alone; the last step is taken below
        z = beta[0] * s * s
        g2, g3 = s * s * _plain_horner(_C2, z), s ** 3 * _plain_horner(_C3, z)
        r = r0[0] * (1 - beta[0] * g2) + eta[0] * (s - beta[0] * g3) + k[0] * g2
        step = (r0[0] * s + eta[0] * g2 + zeta[0] * g3 - h[0]) / r
        s = s - step
        if np.all(np.abs(step) <= 1e-12 * np.abs(s)):
            break

    def g23(sd):
        z = _mul(beta, _mul(sd, sd))
        p2, d2 = _horner(_C2, z[0])
        p3, d3 = _horner(_C3, z[0])
        ss = _mul(sd, sd)
        return _mul(ss, _func(z, p2, d2)), _mul(_mul(ss, sd), _func(z, p3, d3))

    fixed = np.zeros_like(r0)
    fixed[0] = s
    g2, g3 = g23(fixed)
    sd = fixed - (_mul(r0, fixed) + _mul(eta, g2) + _mul(zeta, g3) - h) / r
    g2, g3 = g23(sd)
    g1 = sd - _mul(beta, g3)
    r = r0 - _mul(_mul(r0, beta), g2) + _mul(eta, g1) + _mul(k, g2)
    kr, kr0 = _mul(k, _inv(r)), _mul(k, r0inv)
    fm1, fdot, gdm1 = -_mul(kr0, g2), -_mul(_mul(kr, r0inv), g1), -_mul(kr, g2)
    if drift_first:
        return _mul(fm1, xd) - _mul(_mul(k, g3), v), _mul(fdot, xd) + _mul(gdm1, v)
    return (_mul(fm1 - _mul(h, fdot), x) - _mul(_mul(k, g3) + _mul(h, gdm1), v),
            _mul(fdot, x) + _mul(gdm1, v))


def _levels(pairs):
    """Pairs in sweep order as index arrays: those of one i + j share no body, and each body meets them in order."""
    return [([i for i, j in pairs if i + j == q], [j for i, j in pairs if i + j == q])
            for q in sorted({i + j for i, j in pairs})]


def _pull(x, i, j):
    """G r_ij / r^3"""
    r = x[:, i] - x[:, j]
    r1inv = _inv(_sqrt(_dot(r, r)))
    return GNEWT * _mul(r, _mul(r1inv, _mul(r1inv, r1inv)))


def _kick(x, v, m, h, levels):
    for i, j in levels:
        f = _mul(h, _pull(x, i, j))
        v[:, i] -= _mul(m[:, j], f)
        v[:, j] += _mul(m[:, i], f)


def _correct(x, v, m, h, levels, coeff, with_mass):
    acc = np.zeros_like(x)
    for i, j in levels:
        f = _pull(x, i, j)
        acc[:, i] -= _mul(m[:, j], f)
        acc[:, j] += _mul(m[:, i], f)
    scale = coeff * GNEWT * _mul(h, _mul(h, h))
    for i, j in levels:
        r, a = x[:, i] - x[:, j], acc[:, i] - acc[:, j]
        r2 = _dot(r, r)
        r1inv = _inv(_sqrt(r2))
        r2inv = _mul(r1inv, r1inv)
        along = 3 * _dot(a, r)
        if with_mass:
            along = along + 2 * GNEWT * _mul(m[:, i] + m[:, j], r1inv)
        f = _mul(_mul(scale, _mul(r1inv, _mul(r2inv, r2inv))), _mul(r, along) - _mul(r2, a))
        v[:, i] += _mul(m[:, j], f)
        v[:, j] -= _mul(m[:, i], f)


def _step(x, v, m, h, kick):
    """One AHL21 step of (x, v) in place; kick: the planet pairs take kicks, the others Kepler drifts."""
    n = x.shape[1]
    every = [(i, j) for i in range(n - 1) for j in range(i + 1, n)]
    kicked = _levels([p for p in every if kick and p[0] > 0])
    solved = _levels([p for p in every if not (kick and p[0] > 0)])
    h2 = 0.5 * h

    def solve(levels, drift_first):
        for i, j in levels:
            mij = _inv(m[:, i] + m[:, j])
            k = GNEWT * (m[:, i] + m[:, j])
            dx, dv = _kepler(x[:, i] - x[:, j], v[:, i] - v[:, j], k, h2, drift_first)
            wi, wj = _mul(m[:, j], mij), _mul(m[:, i], mij)
            x[:, i] += _mul(wi, dx)
            v[:, i] += _mul(wi, dv)
            x[:, j] -= _mul(wj, dx)
            v[:, j] -= _mul(wj, dv)

    _kick(x, v, m, h / 6.0, kicked)
    x += _mul(h2, v)
    solve(solved, True)
    if kicked:
        _kick(x, v, m, 2.0 * h / 3.0, kicked)
        _correct(x, v, m, h, kicked, 1.0 / 36.0, False)
    _correct(x, v, m, h, solved, 1.0 / 24.0, True)
    solve(solved[::-1], False)
    x += _mul(h2, v)
    _kick(x, v, m, h / 6.0, kicked)


def _duals(x, v, m, full):
    """Dual (x, v, m) of systems x, v (S, 3, n), m (S, n): derivatives with respect to 7n initial values and, in
    the last place, the step; only the step's without `full`."""
    S, _, n = x.shape
    c = 7 * n if full else 0
    X, V, Mm = np.zeros((2 + c, n, 3, S)), np.zeros((2 + c, n, 3, S)), np.zeros((2 + c, n, 1, S))
    X[0], V[0], Mm[0, :, 0] = x.transpose(2, 1, 0), v.transpose(2, 1, 0), m.T
    if full:
        for b in range(n):
            for q in range(3):
                X[1 + 7 * b + q, b, q] = 1.0
                V[1 + 7 * b + 3 + q, b, q] = 1.0
            Mm[1 + 7 * b + 6, b] = 1.0
    return X, V, Mm


def _step_of(h, like):
    """The step as a dual number whose derivative is the last one."""
    d = np.zeros((like.shape[0], 1, 1, like.shape[3]))
    d[0], d[-1] = h, 1.0
    return d


def _sky(X, V, b):
    return _mul(X[:, 0, :2] - X[:, b, :2], V[:, 0, :2] - V[:, b, :2]).sum(axis=1)


def _integrate(x, v, m, h, steps, full, kick=False, transits=False, last=None, each=None):
    """steps[s] steps of h[s] for each system of one body count; `last`: the length of one step more.

    Returns (X, V, dqdt, events): the duals at each system's end, the last step's derivative by its length, and
    for each transit (system, body, index, start time of the search, its estimate, the duals it starts from)."""
    X, V, M = _duals(x, v, m, full)
    n, S = X.shape[1], X.shape[3]
    h, steps = np.asarray(h, float), np.asarray(steps)
    before = np.array([_sky(X[:1], V[:1], b)[0] for b in range(n)])
    seen, events, dqdt = np.zeros((n, S), int), [], np.zeros((S, 7 * n))
    total = int(steps.max()) + (last is not None)
    for k in range(total):
        on = np.nonzero(steps + (last is not None) > k)[0]
        every = len(on) == S
        x1, v1, m1 = (X, V, M) if every else (X[..., on].copy(), V[..., on].copy(), M[..., on])
        if each is not None:
            each(k, x1, v1)
        x1[-1], v1[-1] = 0.0, 0.0  # the derivative by the step is this step's own
        _step(x1, v1, m1, _step_of(h[on] if k < steps.max() else last, x1), kick)
        if not every:
            X[..., on], V[..., on] = x1, v1
        for b in range(1, n) if transits else ():
            g = _sky(x1[:1], v1[:1], b)[0]
            r = np.sqrt((x1[0, b] ** 2).sum(axis=0))
            for q in np.nonzero((g > 0) & (before[b, on] < 0) & (-x1[0, b, 2] > 0.25 * r))[0]:
                s = on[q]
                events.append((s, b, seen[b, s], (k + 1) * h[s], -g[q] * h[s] / (g[q] - before[b, s]),
                               x1[..., q].copy(), v1[..., q].copy(), m1[..., q].copy()))
                seen[b, s] += 1
            before[b, on] = g
    for b in range(n):
        for q in range(3):
            dqdt[:, 7 * b + q], dqdt[:, 7 * b + 3 + q] = X[-1, b, q], V[-1, b, q]
    return X, V, dqdt, events


def _transit_values(events, full, kick):
    """Per transit: (t, v_sky, b_sky^2) and with `full` their derivatives (3, 7n) as TransitParameters holds them."""
    if not events:
        return np.zeros((0, 3)), np.zeros((0, 3, 0))
    body, t0, dt = np.array([e[1] for e in events]), np.array([e[3] for e in events]), np.array([e[4] for e in events])
    X0, V0, M0 = (np.stack([e[q] for e in events], axis=-1) for q in (5, 6, 7))

    def after(dt, rows):
        X, V, M = X0[rows].copy(), V0[rows].copy(), M0[rows].copy()
        X[-1], V[-1] = 0.0, 0.0
        _step(X, V, M, _step_of(dt, X), kick)
        at = np.arange(len(dt))
        dx = X[:, 0, :2] - X[:, body, :2, at].transpose(1, 2, 0)
        dv = V[:, 0, :2] - V[:, body, :2, at].transpose(1, 2, 0)
        return dx, dv

    few = [0, -1]
    for _ in range(8):
        dx, dv = after(dt, few)
        g = _mul(dx, dv).sum(axis=1)
        dt = dt - g[0] / g[1]
    dx, dv = after(dt, slice(None) if full else few)
    speed = np.sqrt((dv[0] ** 2).sum(axis=0))
    values = np.stack([t0 + dt, speed, (dx[0] ** 2).sum(axis=0)], axis=1)
    g = _mul(dx, dv).sum(axis=1)
    d_t = -g[1:-1] / g[-1]
    d_v = ((dv[0] * dv[1:-1]).sum(axis=1) + (dv[0] * dv[-1]).sum(axis=0) * d_t) / speed
    d_b = 2 * (dx[0] * dx[1:-1]).sum(axis=1)
    return values, np.stack([d_t, d_v, d_b]).transpose(2, 0, 1)


def _jacobian(X, V, s):
    """jac_step of system s from its duals."""
    n = X.shape[1]
    J = np.zeros((7 * n, 7 * n))
    for b in range(n):
        J[7 * b:7 * b + 3] = X[1:-1, b, :, s].T
        J[7 * b + 3:7 * b + 6] = V[1:-1, b, :, s].T
        J[7 * b + 6, 7 * b + 6] = 1.0
    return J


def _seconds(case, full):
    """About how long exact() takes."""
    count, mixed = case.get("systems", 1), case["kind"] in ("host", "serve")
    total = 0.0
    for n in (range(2, case["n"] + 1) if mixed else [case["n"]]):
        share = count / (case["n"] - 1) if mixed else count
        total += case["steps"] * (2 * (2 * n - 3) * 9e-4 + n * (n - 1) * 4e-7 * share * (2 + 7 * n * full))
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "init":
        return _exact_init(case, seed)
    kick, grad = bool(case.get("kick")), bool(case.get("grad", True))
    # a kick group's Jacobian leaves a product of two increments out by design, so it is no derivative of the step
    full = grad and not kick and kind != "serve" and _seconds(case, True) < 15
    if not full and _seconds(case, False) > 15:
        return None
    big = kind == "device" and case["systems"] * case["steps"] > 2e5
    if kind in ("device", "host"):
        b = _filled_batch(case, seed)
        n_of, h_of, steps_of = b.n, b.h, np.rint(b.tmax / b.h).astype(int)
        inputs = [(b.view("x", s).reshape((3, n), order="F"), b.view("v", s).reshape((3, n), order="F"),
                   b.view("m", s)) for s, n in enumerate(b.n)]
        jac_init = [b.view("jac_init", s).reshape((7 * n, 7 * n), order="F") for s, n in enumerate(b.n)]
        ntt = list(b.ntt)
    else:
        st = _states(case, seed)
        n_of, h_of, steps_of = [s.n for s, _, _, _ in st], [h for _, _, h, _ in st], [k for _, _, _, k in st]
        inputs, jac_init = [(s.x, s.v, s.m) for s, _, _, _ in st], [s.jac_init for s, _, _, _ in st]
        ntt = [_ntt(k) for _, _, _, k in st]
    timed = kind not in ("steps", "time", "cartesian") and not big
    found = [None] * len(n_of)
    traj = []
    each = (lambda k, X, V: traj.append((X[..., 0].copy(), V[..., 0].copy()))) if kind == "cartesian" else None
    for n in sorted(set(int(q) for q in n_of)):
        own = [s for s, q in enumerate(n_of) if q == n]
        h = np.array([h_of[s] for s in own])
        steps = np.array([steps_of[s] for s in own])
        last = None
        if kind == "time":
            span = _span(case, h[0], int(steps[0]))
            steps = np.rint(span / h).astype(int)
            last = span - h[0] * steps[0]
        X, V, dqdt, events = _integrate(*(np.stack([inputs[s][q] for s in own]) for q in range(3)), h, steps, full,
                                        kick, timed, last, each)
        values, slopes = _transit_values(events, full, kick)
        for q, s in enumerate(own):
            rows, N = (3 if kind == "parameters" else 1), n
            out = np.zeros((rows, N, ntt[s]))
            dq0 = np.zeros((rows, N, ntt[s], 7, N))
            for e, ev in enumerate(events):
                if ev[0] == q:
                    out[:, ev[1], ev[2]] = values[e, :rows]
                    if full:
                        dq0[:, ev[1], ev[2]] = slopes[e, :rows].reshape((rows, N, 7)).transpose(0, 2, 1)
            del_ = np.einsum("rjckp,pkx->rjcx", dq0, jac_init[s].reshape((N, 7, 7 * N))) if full else None
            if full:
                del_ = del_.reshape((rows, N, ntt[s], N, 7)).transpose(0, 1, 2, 4, 3)
            found[s] = {"x": X[0, :, :, q].T, "v": V[0, :, :, q].T, "out": out, "dq0": dq0, "del": del_,
                        "dqdt": dqdt[q], "jac": _jacobian(X, V, q) if full else None}
    flat = lambda key: np.concatenate([f[key].ravel(order="F") for f in found])  # noqa: E731
    if kind in ("device", "host", "serve"):
        got = {"x": flat("x"), "v": flat("v"), "tt": flat("out") if timed else None, "count": None}
        if kind != "serve":
            got.update(t=None, status=None)
        if grad:
            got.update(jac_step=flat("jac") if full else None, dqdt=flat("dqdt") if kind != "serve" else None,
                       dtdq0=flat("dq0") if full and timed else None,
                       dtdelements=flat("del") if full and timed else None)
        return got
    f = found[0]
    got = {"t": None, "x": f["x"], "v": f["v"]}
    if grad:
        got.update(jac_step=f["jac"], dqdt=f["dqdt"])
    if kind == "transits":
        got.update(tt=f["out"][0], count=None)
        if grad:
            got.update(dtdq0=f["dq0"][0] if full else None, dtdelements=f["del"][0] if full else None)
    elif kind == "parameters":
        got.update(ttbv=f["out"], count=None)
        if grad:
            got.update(dtbvdq0=f["dq0"] if full else None, dtbvdelements=f["del"] if full else None)
    elif kind == "cartesian":
        got.update(out_t=None, out_x=np.stack([X[0].T for X, _ in traj]), out_v=np.stack([V[0].T for _, V in traj]),
                   out_jac=np.stack([_jacobian(X[..., None], V[..., None], 0) for X, V in traj]) if full else None)
    return got


def _exact_init(case, seed):
    """Positions, velocities and their derivatives by the elements: each planet on a Kepler orbit about the
    barycentre of the bodies inside it, at time 0."""
    els = np.stack([el for el, _, _ in _elements(case, seed)])  # S, n, 7: m, P, t0, e cos w, e sin w, I, Omega
    S, n, _ = els.shape
    C = 1 + 7 * n

    def var(b, q, place):
        d = np.zeros((C, S))
        d[0], d[1 + 7 * b + place] = els[:, b, q], 1.0
        return d

    def const(c):
        d = np.zeros((C, S))
        d[0] = c
        return d

    sin = lambda a: _func(a, np.sin(a[0]), np.cos(a[0]))  # noqa: E731
    cos = lambda a: _func(a, np.cos(a[0]), -np.sin(a[0]))  # noqa: E731
    m = [var(b, 0, 6) for b in range(n)]
    inside, rel = m[0], []
    for b in range(1, n):
        P, t0, ec, es, inc, om = (var(b, 1 + q, q) for q in range(6))
        outside = inside + m[b]
        freq = 2 * math.pi * _inv(P)
        cube = GNEWT / (4 * math.pi ** 2) * _mul(outside, _mul(P, P))
        root = np.cbrt(cube[0])
        semi = _func(cube, root, root / (3 * cube[0]))
        ecc = _sqrt(_mul(ec, ec) + _mul(es, es))
        cw, sw = _mul(ec, _inv(ecc)), _mul(es, _inv(ecc))
        flat = _sqrt(const(1.0) - _mul(ecc, ecc))
        # mean anomaly at mid-transit, where true anomaly + w = -pi/2: sin f = -cos w, cos f = -sin w
        down = _inv(const(1.0) - _mul(ecc, sw))
        sE, cE = -_mul(_mul(flat, cw), down), _mul(ecc - sw, down)
        E = cE[0] * sE - sE[0] * cE
        E[0] = np.arctan2(sE[0], cE[0])
        mean = E - _mul(ecc, sE) - _mul(freq, t0)
        F = mean[0] + ecc[0] * np.sin(mean[0])
        for _ in range(30):
            F = F - (F - ecc[0] * np.sin(F) - mean[0]) / (1 - ecc[0] * np.cos(F))
        E = const(F) - (const(F) - np.sin(F) * ecc - mean) / (1 - ecc[0] * np.cos(F))
        cE, sE = cos(E), sin(E)
        px, py = _mul(semi, cE - ecc), _mul(semi, _mul(flat, sE))
        rate = _mul(_mul(freq, semi), _inv(const(1.0) - _mul(ecc, cE)))
        vx, vy = -_mul(rate, sE), _mul(rate, _mul(flat, cE))
        ci, si, co, so = cos(inc), sin(inc), cos(om), sin(om)
        both = []
        for a, c in ((px, py), (vx, vy)):
            a, c = _mul(cw, a) - _mul(sw, c), _mul(sw, a) + _mul(cw, c)
            c, z = _mul(ci, c), _mul(si, c)
            both.append(np.stack([_mul(co, a) - _mul(so, c), _mul(so, a) + _mul(co, c), z], axis=1))
        rel.append((both, _mul(m[b], _inv(outside))))
        inside = outside
    pos = [[None] * n, [None] * n]
    for q in (0, 1):
        centre = np.zeros((C, 3, S))
        for b in range(n - 1, 0, -1):
            centre = centre - _mul(rel[b - 1][1][:, None], rel[b - 1][0][q])
            pos[q][b] = centre + rel[b - 1][0][q]
        pos[q][0] = centre
    x, v = (np.stack(pos[q], axis=1) for q in (0, 1))  # C, n, 3, S
    jac = np.zeros((S, 7 * n, 7 * n))
    for b in range(n):
        jac[:, 7 * b:7 * b + 3] = x[1:, b].transpose(2, 1, 0)
        jac[:, 7 * b + 3:7 * b + 6] = v[1:, b].transpose(2, 1, 0)
        jac[:, 7 * b + 6, 7 * b + 6] = 1.0
    return {"x": x[0].transpose(2, 1, 0), "v": v[0].transpose(2, 1, 0), "jac_init": jac}
