"""What is measured: the work that users of the library have it do, through its public entry points.

The workloads are the library's own: the cold uniform sphere of the reference's input (unit radius,
c = 1, its dt), and Plummer spheres with a black hole (BH) of 1 % of the stellar mass in Henon units
(softening 0.04 / N^(1/3), dt = 1/1024, c = 1000), at the sizes of its configurations, tests and
benchmark, in both precisions.  FP64 is the default of every entry point and the parity mode; the
mixed precision (FP32 pair terms) is what large integrations, ensembles and fits run in.

Kinds of call:
  dropin    the reference's force(): host arrays in and out, one evaluation
  device    one evaluation on the caller's own device arrays and stream
  steps     a device-resident context advanced by some steps, state read back (a run between snapshots)
  loop      one pass of the command-line driver's loop: the energy owed at a snapshot, fused into
            the steps that follow it, and the state for the next snapshot
  energy    the energies of a state
  ensemble  many clusters advanced together, states read back
  vjp       the vector-Jacobian product of one force evaluation
  gradient  one iteration of a fit: initial state in, steps forward, gradient of a loss back
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

import pn_gb300 as pn

F64, MIXED = "f64", "mixed"
PAIR_FLOPS = 55.0    # one ordered star pair of the 1PN force, its shared terms formed once for both stars
ENERGY_FLOPS = 30.0  # the same of the energy sums
VJP_FLOPS = 140.0    # the same of the force's vector-Jacobian product


def listed():
    return [
        # a few hundred stars: launch-bound runs (the size of the smoke test and the ABI tests)
        {"name": "steps_f64_256", "kind": "steps", "prec": F64, "model": "plummer", "n": 257, "k": 16},
        # a caller's own loop around the reference's force(), small system
        {"name": "dropin_force_1k", "kind": "dropin", "prec": F64, "model": "sphere", "n": 1001},
        # a framework that holds its state in device memory, odd size
        {"name": "device_force_2k", "kind": "device", "prec": F64, "model": "plummer", "n": 2050},
        # the driver's loop between two snapshots, a medium system
        {"name": "loop_f64_4k", "kind": "loop", "prec": F64, "model": "sphere", "n": 4097, "k": 4},
        # the reference's own run: 10,000 stars + BH
        {"name": "steps_f64_10k", "kind": "steps", "prec": F64, "model": "sphere", "n": 10001, "k": 2},
        # the energy of a state (initial_energy, snapshots written with checkpoints)
        {"name": "energy_f64_20k", "kind": "energy", "prec": F64, "model": "plummer", "n": 20001},
        # the largest FP64 configuration, through the reference's entry point
        {"name": "dropin_force_65k", "kind": "dropin", "prec": F64, "model": "plummer", "n": 65537},
        # long mixed-precision runs: a small cluster, a medium one, the headline size
        {"name": "steps_mixed_1k", "kind": "steps", "prec": MIXED, "model": "plummer", "n": 1025, "k": 4},
        {"name": "steps_mixed_16k", "kind": "steps", "prec": MIXED, "model": "plummer", "n": 16385, "k": 4},
        {"name": "steps_mixed_262k", "kind": "steps", "prec": MIXED, "model": "plummer", "n": 262145, "k": 1},
        # parameter studies: many clusters of different sizes at once
        {"name": "ensemble_mixed", "kind": "ensemble", "prec": MIXED, "model": "plummer", "clusters": 48,
         "n": 1024, "nmax": 16384, "k": 1},
        # fitting an initial state, one iteration: the size of the adjoint configuration
        {"name": "gradient_mixed_16k", "kind": "gradient", "prec": MIXED, "model": "plummer", "n": 16385, "k": 4,
         "keep": 2},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dropin", "device", "steps", "steps", "steps", "loop", "energy", "ensemble", "vjp", "gradient"])
    if kind == "dropin":
        return {"kind": kind, "prec": F64, "model": rng.choice(["sphere", "plummer"]), "n": size(200, 50000)}
    if kind == "device":
        return {"kind": kind, "prec": F64, "model": "plummer", "n": size(200, 30000)}
    if kind == "steps":
        prec = rng.choice([F64, MIXED])
        if prec == F64:
            n = size(200, 20000)
            return {"kind": kind, "prec": prec, "model": "plummer", "n": n, "k": 16 if n < 3000 else 4 if n < 10000 else 1}
        n = size(1000, 200000)
        return {"kind": kind, "prec": prec, "model": "plummer", "n": n, "k": 4 if n < 30000 else 1}
    if kind == "loop":
        return {"kind": kind, "prec": F64, "model": "sphere", "n": size(500, 12000), "k": rng.randint(2, 5)}
    if kind == "energy":
        return {"kind": kind, "prec": F64, "model": "plummer", "n": size(300, 40000)}
    if kind == "ensemble":
        return {"kind": kind, "prec": MIXED, "model": "plummer", "clusters": rng.randint(6, 64), "n": 512,
                "nmax": size(2000, 20000), "k": rng.randint(1, 2)}
    if kind == "vjp":
        return {"kind": kind, "prec": F64, "model": "plummer", "n": size(300, 6000)}
    prec = rng.choice([F64, MIXED])
    n = size(300, 6000) if prec == F64 else size(1000, 16000)
    return {"kind": kind, "prec": prec, "model": "plummer", "n": n, "k": rng.randint(2, 4), "keep": 2}


# ------------------------------------------------------------------ inputs
def _iso(rng, r):
    z = 1.0 - 2.0 * rng.random(r.size)
    ph = 2.0 * math.pi * rng.random(r.size)
    s = np.sqrt(1.0 - z * z)
    return np.stack([s * np.cos(ph), s * np.sin(ph), z], 1) * r[:, None]


def _speed(rng, n):
    """q = v / v_escape of a Plummer sphere, density ~ q^2 (1 - q^2)^(7/2) (Aarseth, Henon & Wielen 1974)."""
    q = np.empty(0)
    while q.size < n:
        a, b = rng.random(2 * n + 64), 0.1 * rng.random(2 * n + 64)
        q = np.concatenate([q, a[b < a * a * (1.0 - a * a) ** 3.5]])
    return q[:n]


def _system(model, n, rng):
    """x, v, m with the BH in row 0 at the origin at rest, and the run's eps, dt, inv_c2."""
    ns = n - 1
    x, v, m = np.zeros((n, 3)), np.zeros((n, 3)), np.full(n, 1.0 / ns)
    if model == "sphere":  # cold, unit radius, read from a file of floats as the reference's input is
        x[1:] = _iso(rng, np.cbrt(rng.random(ns))).astype(np.float32)
        m[0] = 100.0 / n
        return x, v, m, 0.001, 1.0 / 131072.0, 1.0
    r = 1.0 / np.sqrt((0.001 + 0.998 * rng.random(ns)) ** (-2.0 / 3.0) - 1.0)
    unit = 3.0 * math.pi / 16.0
    x[1:] = _iso(rng, r) * unit
    v[1:] = _iso(rng, _speed(rng, ns) * math.sqrt(2.0) * (1.0 + r * r) ** -0.25) / math.sqrt(unit)
    x[1:] -= x[1:].mean(0)
    v[1:] -= v[1:].mean(0)
    m[0] = 0.01
    return x, v, m, 0.04 / ns ** (1.0 / 3.0), 1.0 / 1024.0, 1e-6


def _sizes(case):
    """The sizes of an ensemble's clusters, spread over the logarithm of their range."""
    lo, hi, c = case["n"], case["nmax"], case["clusters"]
    return [1 + int(lo * (hi / lo) ** ((i + 0.5) / c)) for i in range(c)]


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "ensemble":
        return [_system(case["model"], n, rng) for n in _sizes(case)]
    x, v, m, eps, dt, c2 = _system(case["model"], case["n"], rng)
    if case["kind"] == "gradient":  # the positions to be fitted: a slightly wider cluster, observed with an error
        extra = 0.01 * x + rng.normal(0.0, 1e-3, x.shape)
    else:
        extra = rng.normal(0.0, 1.0, x.shape)
    return x, v, m, eps, dt, c2, extra


def prepare(case, seed):
    kind, prec = case["kind"], pn.PN_PREC_MIXED if case["prec"] == MIXED else pn.PN_PREC_FP64
    got = _inputs(case, seed)
    if kind == "ensemble":
        sys = [pn.System(x, v, m) for x, v, m, *_ in got]
        ens = pn.Ensemble(sys, [s[3] for s in got], precision=prec, dt=got[0][4], inv_c2=got[0][5])
        return {"kind": kind, "ens": ens, "k": case["k"]}
    x, v, m, eps, dt, c2, extra = got
    if kind == "dropin":
        return {"kind": kind, "x": x, "v": v, "m": m, "eps": eps}
    c = pn.Context(case["n"], precision=prec, eps=eps, dt=dt, inv_c2=c2)
    state = {"kind": kind, "c": c, "n": case["n"], "k": case.get("k", 0)}
    if kind == "device":
        state.update(stream=torch.cuda.Stream(), x=torch.tensor(x, device="cuda"), v=torch.tensor(v, device="cuda"),
                     m=torch.tensor(m, device="cuda"), a=torch.empty(x.shape, dtype=torch.float64, device="cuda"))
        return state
    if kind == "gradient":
        state.update(x=x, v=v, m=m, keep=case["keep"], target=x + extra)
        return state
    c.set_state(x, v, m)
    if kind == "vjp":
        state["abar"] = extra
    return state


def run(state):
    kind = state["kind"]
    if kind == "dropin":
        return pn.force(state["x"], state["v"], state["m"], state["eps"])
    if kind == "ensemble":
        state["ens"].steps(state["k"])
        x, v = state["ens"].get_state()
        return [np.concatenate(x), np.concatenate(v)]
    c = state["c"]
    if kind == "device":
        c.force_device(state["n"], state["x"].data_ptr(), state["v"].data_ptr(), state["m"].data_ptr(),
                       state["a"].data_ptr(), state["stream"].cuda_stream)
        return state["a"]
    if kind == "steps":
        c.steps(state["k"])
        return list(c.get_state())
    if kind == "loop":
        e = c.steps_energy(state["k"])
        return [np.array(e)] + list(c.get_state())
    if kind == "energy":
        return np.array(c.energy())
    if kind == "vjp":
        xb, vb, m0b = c.force_vjp(state["abar"])
        return [xb, vb, np.float64(m0b)]
    c.set_state(state["x"], state["v"], state["m"])
    c.adjoint_forward(state["k"], state["keep"])
    xT, vT = c.get_state()
    x0b, v0b, m0b = c.adjoint_backward(2.0 * (xT - state["target"]), np.zeros_like(vT))
    return [xT, vT, x0b, v0b, np.float64(m0b)]


def work(case):
    kind, k = case["kind"], case.get("k", 1)
    if kind == "ensemble":
        ns = _sizes(case)
        return {"bytes": 104.0 * sum(ns), "flops": 3.0 * k * PAIR_FLOPS * sum(float(n) * n for n in ns)}
    n = float(case["n"])
    pairs = n * n
    if kind in ("dropin", "device"):
        return {"bytes": 80.0 * n, "flops": PAIR_FLOPS * pairs}
    if kind == "steps":
        return {"bytes": 104.0 * n, "flops": 3.0 * k * PAIR_FLOPS * pairs}
    if kind == "loop":
        return {"bytes": 104.0 * n + 32.0, "flops": (3.0 * k * PAIR_FLOPS + 6.0) * pairs}
    if kind == "energy":
        return {"bytes": 56.0 * n + 32.0, "flops": ENERGY_FLOPS * pairs}
    if kind == "vjp":
        return {"bytes": 128.0 * n, "flops": (PAIR_FLOPS + VJP_FLOPS) * pairs}
    # forward steps, and the reversal; steps before the last kept state are run twice
    again = max(0, k - case["keep"])
    return {"bytes": 200.0 * n, "flops": 3.0 * pairs * ((k + again) * PAIR_FLOPS + k * VJP_FLOPS)}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
def _force(x, v, m, eps, c2, rows=None):
    """The accelerations of all particles (G = 1): softened Newtonian forces, the 1PN terms of the BH
    and the stars and the three-body cross terms weighted by c2, from sums over all star pairs (the
    pair of a star with itself among them, as the reference's loops have it, and its own removal of
    that pair).  Differentiable; evaluated by blocks of rows."""
    s, vs, mu, m0, e2 = x[1:] - x[0], v[1:], m[1:], m[0], eps * eps
    q = (s * s).sum(1)
    R = (q + e2) ** -0.5
    R3 = R ** 3
    mr3 = mu * R3

    def sums(si, vi, qi):
        d = s[None] - si[:, None]
        rho = (d * d).sum(2) + e2
        Q = rho ** -0.5
        Q3 = Q / rho
        mq3 = mu * Q3
        G = (mq3[..., None] * d).sum(1)
        phi, s0, u = (mu * Q).sum(1), mq3.sum(1), (mr3 * Q).sum(1)
        vjd, vid = (vs[None] * d).sum(2), (vi[:, None] * d).sum(2)
        dv = vs[None] - vi[:, None]
        br = (1.25 * m0 * R + 0.25 * m0 * R3 * (rho - qi[:, None] - e2) + (vi * vi).sum(1)[:, None]
              - 2.0 * (dv * dv).sum(2) + 1.5 * vjd * vjd / rho)
        cd, cv = mq3 * br + 3.5 * m0 * mr3 * Q, mq3 * (4.0 * vid - 3.0 * vjd)
        W = (cd[..., None] * d + cv[..., None] * dv).sum(1)
        return torch.cat([G, phi[:, None], s0[:, None], u[:, None], W], 1)

    rows = rows or max(1, (1 << 25) // s.shape[0])
    parts = []
    for i in range(0, s.shape[0], rows):
        blk = (s[i:i + rows], vs[i:i + rows], q[i:i + rows])
        if torch.is_grad_enabled() and s.requires_grad:
            parts.append(torch.utils.checkpoint.checkpoint(sums, *blk, use_reentrant=False))
        else:
            parts.append(sums(*blk))
    S = torch.cat(parts)
    G, phi, s0, u, W = S[:, 0:3], S[:, 3], S[:, 4], S[:, 5], S[:, 6:9]
    a1, b3, c3, mom = (mu * R).sum(), (mr3[:, None] * s).sum(0), (mr3 * q).sum(), (mu[:, None] * vs).sum(0)
    v2, vsd = (vs * vs).sum(1), (vs * s).sum(1)
    vp, ps, sb, sg = vs @ mom, s @ mom, s @ b3, (s * G).sum(1)
    cs = (-m0 * R3 * (4 * m0 * R - v2) + 5 * m0 * mr3 * R - 4 * mr3 * v2
          - m0 * R3 * (4 * phi + 1.25 * a1 - 0.25 * c3 + 0.5 * sb) + 3.5 * m0 * u + 4 * R3 * vp
          + mr3 * m0 * (4 / eps + 1.25 * R + 0.25 * q * R3) - 3.5 * mr3 * m0 * (1 / eps - R) - 4 * mr3 * v2)
    cv = -4 * m0 * R3 * vsd + 14 * mr3 * vsd - 3 * R3 * ps
    star = (cs[:, None] * s + cv[:, None] * vs + (4 * m0 * R)[:, None] * G - (3.5 * m0 * R)[:, None] * b3
            - (4 * R3 * vsd)[:, None] * mom + W)
    bs = (mr3 * (5 * m0 * R - 2 * v2 + 1.5 * vsd * vsd / q) + 4 * mr3 * R * mu
          + mr3 * (4 * a1 + 1.25 * phi + 0.25 * (-2 * sg - (phi - e2 * s0))) - 4 * mr3 / m0 * vp
          + mr3 * mu * (4 * R + 1.25 * eps) - 4 * mr3 * mu / m0 * v2)
    bv = 3 * mr3 * vsd + 4 * mr3 / m0 * ps + 7 * mr3 * mu / m0 * vsd
    bh = (bs[:, None] * s + bv[:, None] * vs - (3.5 * R * mu)[:, None] * G + (3 * mr3 / m0 * vsd)[:, None] * mom).sum(0)
    return torch.cat([(b3 + c2 * bh)[None], G - (m0 * R3)[:, None] * s + c2 * star])


def _step(x, v, m, eps, dt, c2):
    """One step of the reference's three-evaluation scheme."""
    x1, v1 = x + 0.5 * dt * v, v + 0.5 * dt * _force(x, v, m, eps, c2)
    x2, v2 = x + 0.5 * dt * v1, v + 0.5 * dt * _force(x1, v1, m, eps, c2)
    x3, v3 = x + dt * v2, v + dt * _force(x2, v2, m, eps, c2)
    return (x + 2 * x1 + 2 * x2 + x3) / 6, (v + 2 * v1 + 2 * v2 + v3) / 6


def _energy(x, v, m, eps, c2):
    s, vs, mu, m0, e2 = x[1:] - x[0], v[1:], m[1:], m[0], eps * eps
    R = ((s * s).sum(1) + e2) ** -0.5
    phi, psi = torch.empty_like(R), torch.empty_like(R)
    rows = max(1, (1 << 25) // s.shape[0])
    for i in range(0, s.shape[0], rows):
        d = s[None] - s[i:i + rows, None]
        Q = ((d * d).sum(2) + e2) ** -0.5
        vi = vs[i:i + rows]
        t = 7 * (vi @ vs.T) + (vi[:, None] * d).sum(2) * (vs[None] * d).sum(2) * Q * Q
        phi[i:i + rows], psi[i:i + rows] = (mu * Q).sum(1), (mu * Q * t).sum(1)
    v2, v0 = (vs * vs).sum(1), v[0]
    mr, a1 = m0 * R, (mu * R).sum()
    kin = 0.5 * ((mu * v2).sum() + m0 * (v0 * v0).sum())
    pot = 0.5 * ((mu * (mu / eps - mr - phi)).sum() - m0 * a1)
    one = (mu * (0.375 * v2 * v2 + 1.5 * mr * v2 + 0.5 * mr * mr
                 + 0.5 * mr * (3 * v2 - 7 * (vs @ v0) - (s @ v0) * (s * vs).sum(1) * R * R))).sum()
    two = (0.25 * mu * (6 * v2 * phi - psi) + m0 * mu * R * phi + 0.5 * m0 * mu * R * a1
           + 0.25 * mu * mu / eps * v2 - m0 * mu * mu * (R / eps + 0.5 * R * R)).sum()
    return torch.stack([pot, kin, c2 * one, kin + pot + c2 * (one + two)])


def exact(case, seed):
    kind, k = case["kind"], case.get("k", 0)
    if kind != "ensemble" and float(case["n"]) ** 2 * max(1, 3 * k) > 3e10:
        return None
    got = _inputs(case, seed)

    def t(a):
        return torch.tensor(a, dtype=torch.float64, device="cuda")

    with torch.set_grad_enabled(kind in ("vjp", "gradient")):
        if kind == "ensemble":
            xs, vs = [], []
            for x, v, m, eps, dt, c2 in got:
                x, v, m = t(x), t(v), t(m)
                for _ in range(k):
                    x, v = _step(x, v, m, eps, dt, c2)
                xs.append(x)
                vs.append(v)
            return [torch.cat(xs), torch.cat(vs)]
        x, v, m, eps, dt, c2, extra = got
        x, v, m = t(x), t(v), t(m)
        if kind == "dropin":
            return _force(x, v, m, eps, 1.0)
        if kind == "device":
            return _force(x, v, m, eps, c2)
        if kind == "energy":
            return _energy(x, v, m, eps, c2)
        if kind in ("steps", "loop"):
            out = [_energy(x, v, m, eps, c2)] if kind == "loop" else []
            for _ in range(k):
                x, v = _step(x, v, m, eps, dt, c2)
            return out + [x, v]
        x.requires_grad_()
        v.requires_grad_()
        m.requires_grad_()
        if kind == "vjp":
            gx, gv, gm = torch.autograd.grad((_force(x, v, m, eps, c2) * t(extra)).sum(), (x, v, m))
            return [gx, gv, gm[0]]
        xT, vT = x, v
        for _ in range(k):
            xT, vT = _step(xT, vT, m, eps, dt, c2)
        gx, gv, gm = torch.autograd.grad(((xT - (t(got[0]) + t(extra))) ** 2).sum(), (x, v, m))
        return [xT.detach(), vT.detach(), gx, gv, gm[0]]
