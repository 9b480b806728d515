"""Timed cases of the propagation library: what its users have it do, over the
range of systems it takes.

A case is one call of a public entry point of mpc_tdse.Context on one system.

Systems (couplings and energies made from the seed):
  electrons 1: hydrogen-like, one block per l, all about the same size -- 60 to
    400 states per l, l_max 1 to 9 (292 x 6 and 388 x 9 are the kept states of
    300 and 400 B-splines in a box of 200 a.u.; other sizes come from
    `states_in_l`, which users set freely, so blocks are odd and ragged);
  electrons 2: helium-CI-like, three to five dense blocks of 400 to 5000
    states per total L (18,000 states is a 400-B-spline CI).
Both gauges; the start state is one from the middle of a pulse (most of the
population in the ground state, the rest spread over many orders of
magnitude), the field that of a pulse in progress.

Operations:
  rhs       one right-hand side (a user's own integrator calls this)
  step      one RKF78 step at a given field (idem)
  propagate the step loop of the reference's main, one pulse, histories kept
  advance   many pulses of uneven length at once, the reference's fixed step
  adaptive  many pulses at once, each with its own step control
  grad      objective and its adjoint gradient, one pulse
  bgrad     the same for many control sets at once
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "mp-citdse_b200"))
import mpc_tdse  # noqa: E402

# Couplings beyond this size cannot stay on the chip between two products of a
# step (126 MB of L2; registers and shared memory hold about 70 MB).
ON_CHIP = 128e6
PRODUCTS = 12   # of one step: the degree of the step's stability polynomial


def listed():
    return [
        # one right-hand side of a 1e basis: the smallest call, all latency
        dict(name="rhs-1e", op="rhs", electrons=1, n="292,292,292,292,292,292", gauge="l"),
        # one RKF78 step of a small two-electron basis with ragged blocks
        dict(name="step-2e", op="step", electrons=2, n="1031,1207,1500,1333", gauge="v", dt=0.1),
        # the plain hydrogen run (300 B-splines, l_max 5), a piece of its loop
        dict(name="prop-1e", op="propagate", electrons=1, n="292,292,292,292,292,292", gauge="l",
             shape="sine", dt=0.1, steps=400),
        # the larger hydrogen basis (400 B-splines, l_max 8), velocity gauge, ragged
        dict(name="prop-1e-lmax8", op="propagate", electrons=1,
             n="388,388,387,387,386,386,385,385,384", gauge="v", shape="sine", dt=0.05, steps=300),
        # a small helium basis: couplings of 52 MB
        dict(name="prop-2e-small", op="propagate", electrons=2, n="1201,1407,1603,1501",
             gauge="v", shape="gaussian", dt=0.1, steps=150),
        # the helium CI run: couplings of 491 MB
        dict(name="prop-2e", op="propagate", electrons=2, n="3983,4411,4702,4904", gauge="v",
             shape="sine", dt=0.1, steps=60),
        # a scan over pulse parameters on the plain hydrogen basis
        dict(name="advance-1e-256", op="advance", electrons=1, n="292,292,292,292,292,292",
             gauge="l", shape="sine", dt=0.05, pulses=256, steps=160),
        # the tail of a scan, or a small one: few pulses at once
        dict(name="advance-1e-6", op="advance", electrons=1, n="292,292,292,292,292,292",
             gauge="l", shape="sine", dt=0.05, pulses=6, steps=200),
        # a scan on a helium basis
        dict(name="advance-2e-64", op="advance", electrons=2, n="2101,2407,2603,2501,2302",
             gauge="v", shape="sine", dt=0.1, pulses=64, steps=16),
        # adaptive steps, pulses of uneven length
        dict(name="adaptive-1e-48", op="adaptive", electrons=1, n="292,292,292,292,292,292",
             gauge="l", shape="sine", pulses=48, window=2.5),
        # the gradient of the ionisation yield in the larger hydrogen basis
        dict(name="grad-1e-lmax8", op="grad", electrons=1,
             n="388,388,388,388,388,388,388,388,388", gauge="l", shape="sine", dt=0.05,
             steps=192, controls=1024),
        # the same for many control sets at once
        dict(name="bgrad-1e-48", op="bgrad", electrons=1, n="292,292,292,292,292,292",
             gauge="l", shape="sine", dt=0.05, steps=96, controls=256, pulses=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["rhs", "step", "propagate", "propagate", "advance", "advance", "adaptive",
                     "grad", "bgrad"])
    electrons = 1 if op in ("adaptive", "grad", "bgrad") else rng.choice([1, 2])
    if electrons == 1:
        base, blocks = _log(rng, 60, 400), rng.randint(2, 10)
        n = [max(40, base - rng.randint(0, max(1, base // 20))) for _ in range(blocks)]
    else:
        base, blocks = _log(rng, 400, 4000), rng.randint(3, 5)
        n = [int(base * rng.uniform(0.8, 1.25)) for _ in range(blocks)]
    case = dict(op=op, electrons=electrons, n=",".join(map(str, n)), gauge=rng.choice("lv"))
    if op == "rhs":
        return case
    if op != "adaptive":
        case["dt"] = rng.choice([0.05, 0.1])
    if op == "step":
        return case
    case["shape"] = rng.choice(["sine", "sine", "gaussian"])
    if op in ("advance", "adaptive", "bgrad"):
        case["pulses"] = _log(rng, 2, 256) if electrons == 1 else _log(rng, 4, 64)
    if op == "adaptive":
        case["pulses"] = min(case["pulses"], 96)
        case["window"] = round(rng.uniform(1.0, 3.0), 3)
    else:
        case["steps"] = _log(rng, 20, 400)
    if op in ("grad", "bgrad"):
        case["controls"] = _log(rng, 16, 1024)
        case["steps"] = min(case["steps"], 192)
    if op == "bgrad":
        case["pulses"] = min(case["pulses"], 64)
    # no more than the largest listed case
    top = max(work(c)["flops"] for c in listed())
    while work(case)["flops"] > top:
        k = "steps" if case.get("steps", 0) > 8 else "pulses" if case.get("pulses", 0) > 4 \
            else "window"
        case[k] = case[k] // 2 if k != "window" else case[k] / 2
    return case


def _sizes(case):
    return [int(v) for v in case["n"].split(",")]


def _batch(case):
    return case.get("pulses", 1)


def _step_counts(case):
    """Steps of each pulse of a scan: uneven, the longest has `steps`."""
    B = _batch(case)
    return [max(1, int(case["steps"] * (0.4 + 0.6 * ((7 * b) % B + 1) / B))) for b in range(B)]


def work(case):
    n = _sizes(case)
    S, ntot, B = sum(a * b for a, b in zip(n, n[1:])), sum(n), _batch(case)
    product = 8.0 * S + 20.0 * ntot       # one product with the couplings, one pulse
    op = case["op"]
    if op == "rhs":
        passes, flops = 1, product
    elif op == "step":
        passes, flops = PRODUCTS, PRODUCTS * product
    elif op == "propagate":
        passes = PRODUCTS * case["steps"]
        flops = passes * product
    elif op == "advance":
        st = _step_counts(case)
        passes, flops = PRODUCTS * max(st), PRODUCTS * sum(st) * product
    elif op == "adaptive":                # 13 stages; about 0.11 a.u. a step
        st = case["window"] * 0.7 / 0.11
        passes, flops = 13 * st, 13 * st * B * product
    else:                                 # forward, and the transposed products back
        passes = 2 * PRODUCTS * case["steps"]
        flops = passes * B * product
    io = 16.0 * ntot * B * 2
    return {"bytes": (8.0 * S if 8.0 * S < ON_CHIP else 8.0 * S * passes) + io, "flops": flops}


# ---- inputs ---------------------------------------------------------------

def _energies(case, rng):
    n = _sizes(case)
    out = []
    if case["electrons"] == 1:
        # Rydberg levels that fit in the box, then box continuum up to ~11 a.u.
        R = 200.0 * max(n) / 298.0
        for l, k in enumerate(n):
            bound = [-0.5 / (j * j) for j in range(l + 1, 100) if 2 * j * j < 0.5 * R][:k // 4]
            cont = 0.5 * ((np.arange(1, k - len(bound) + 1) + 0.5 * l) * np.pi / R) ** 2
            out.append(np.sort(np.concatenate([bound, cont])))
    else:
        for L, k in enumerate(n):
            nb, ns = max(8, k // 40), k // 2
            bound = -2.0 - 0.9037 * np.exp(-np.arange(nb) / 3.0) * (1.0 if L == 0 else 0.75)
            single = rng.uniform(-2.0, 0.0, ns)
            double = 15.0 * rng.uniform(0.0, 1.0, k - nb - ns) ** 1.5
            out.append(np.sort(np.concatenate([bound, single, double])))
    return out


def _system(case, seed):
    """(energies per block, coupling blocks on the GPU)"""
    E = _energies(case, np.random.default_rng(seed))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    D = []
    for a, b in zip(E, E[1:]):
        m = torch.randn(len(a), len(b), generator=gen, device="cuda", dtype=torch.float64)
        if case["electrons"] == 1:
            ea = torch.as_tensor(a, device="cuda")[:, None]
            eb = torch.as_tensor(b, device="cuda")[None, :]
            m *= (2.0 if case["gauge"] == "l" else 0.5) / (1 + 4 * (ea - eb).abs())
            m /= 1 + ea.clamp(min=0) + eb.clamp(min=0)
        else:
            m *= 0.5 / math.sqrt(len(a) + len(b))
        D.append(m)
    return E, D


def _states(case, seed):
    """Start states [B, size]: mid-pulse, unit norm."""
    rng = np.random.default_rng([seed, 1])
    B, N = _batch(case), sum(_sizes(case))
    x = (rng.standard_normal((B, N)) + 1j * rng.standard_normal((B, N))) \
        * 10.0 ** rng.uniform(-7.0, -2.0, (B, N))
    x[:, 0] += 1.0
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _pulses(case, seed):
    """Parameters of the pulses, in a.u.: (intensity, frequency, CEP, cycles)."""
    rng = np.random.default_rng([seed, 2])
    out = []
    for _ in range(_batch(case)):
        if case["electrons"] == 1:
            I, lam = 10.0 ** rng.uniform(13.0, 14.3), rng.uniform(400.0, 1200.0)
        else:
            I, lam = 10.0 ** rng.uniform(14.0, 14.7), rng.uniform(200.0, 500.0)
        out.append((I / 3.50944e16, 45.563353 / lam, rng.uniform(0.0, 1.0),
                    int(rng.integers(4, 12))))
    return out


def _start_times(case, seed):
    """Times inside the pulses: 20 to 40 % of each one's length; a gradient
    starts with its pulse, whose controls cover the time that it runs."""
    if case["op"] in ("grad", "bgrad"):
        return np.zeros(_batch(case))
    rng = np.random.default_rng([seed, 3])
    return np.array([rng.uniform(0.2, 0.4) * c * 2 * math.pi / w
                     for _, w, _, c in _pulses(case, seed)])


def _windows(case, seed):
    rng = np.random.default_rng([seed, 4])
    return case["window"] * rng.uniform(0.4, 1.0, _batch(case))


def _controls(case, seed):
    rng = np.random.default_rng([seed, 5])
    return 5e-4 * rng.standard_normal((_batch(case), case["controls"]))


def prepare(case, seed):
    E, D = _system(case, seed)
    s = {"case": case, "x": _states(case, seed)}
    dip = np.concatenate([d.cpu().numpy().ravel() for d in D])
    s["ctx"] = mpc_tdse.Context(_sizes(case), np.concatenate(E), dip, case["gauge"])
    if case["op"] in ("rhs", "step"):
        s["F"] = 0.03 + 0.01 * (seed % 7)
        return s
    s["t0"] = _start_times(case, seed)
    s["pulses"] = []
    for I, w, cep, cycles in _pulses(case, seed):
        tau = mpc_tdse.period(w, cycles)
        s["pulses"].append(mpc_tdse.pulse_setup(case["shape"], case["gauge"], I, w, cep, cycles,
                                                tau))
    if case["op"] == "advance":
        s["steps"] = np.array(_step_counts(case))
    if case["op"] == "adaptive":
        s["t_end"] = s["t0"] + _windows(case, seed)
    if case["op"] in ("grad", "bgrad"):
        s["u"] = _controls(case, seed)
        s["T"] = (case["steps"] + 1) * case["dt"]
    return s


def run(s):
    case, ctx, x = s["case"], s["ctx"], s["x"]
    op = case["op"]
    if op == "rhs":
        return ctx.rhs(s["F"], x[0])
    if op == "step":
        return ctx.rk78_step(s["F"], case["dt"], x[0])
    if op == "propagate":
        return ctx.propagate(s["pulses"][0], s["t0"][0], case["dt"], case["steps"], x[0])
    if op == "advance":
        return ctx.batch_advance(s["pulses"], s["t0"], case["dt"], s["steps"], x, history=True)
    if op == "adaptive":
        return ctx.batch_propagate(s["pulses"], s["t0"], s["t_end"], x, dt_max=0.15)
    if op == "grad":
        return ctx.objective_gradient(s["pulses"][0], s["u"][0], s["T"], s["t0"][0], case["dt"],
                                      case["steps"], x[0])
    return ctx.batch_objective_gradient(s["pulses"], s["u"], s["T"], s["t0"][0], case["dt"],
                                        case["steps"], x)


# ---- the same in plain torch, 64 bits ---------------------------------------

class _Tableau:
    """Fehlberg's 7(8) pair (NASA TR R-287, 1968)."""

    def __init__(self):
        A = [[], [2 / 27], [1 / 36, 1 / 12], [1 / 24, 0, 1 / 8], [5 / 12, 0, -25 / 16, 25 / 16],
             [1 / 20, 0, 0, 1 / 4, 1 / 5],
             [-25 / 108, 0, 0, 125 / 108, -65 / 27, 125 / 54],
             [31 / 300, 0, 0, 0, 61 / 225, -2 / 9, 13 / 900],
             [2, 0, 0, -53 / 6, 704 / 45, -107 / 9, 67 / 90, 3],
             [-91 / 108, 0, 0, 23 / 108, -976 / 135, 311 / 54, -19 / 60, 17 / 6, -1 / 12],
             [2383 / 4100, 0, 0, -341 / 164, 4496 / 1025, -301 / 82, 2133 / 4100, 45 / 82,
              45 / 164, 18 / 41],
             [3 / 205, 0, 0, 0, 0, -6 / 41, -3 / 205, -3 / 41, 3 / 41, 6 / 41, 0],
             [-1777 / 4100, 0, 0, -341 / 164, 4496 / 1025, -289 / 82, 2193 / 4100, 51 / 82,
              33 / 164, 12 / 41, 0, 1]]
        self.A = A
        self.C = [0, 2 / 27, 1 / 9, 1 / 6, 5 / 12, 1 / 2, 5 / 6, 1 / 6, 2 / 3, 1 / 3, 1, 0, 1]
        self.B8 = [0, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 0, 41 / 840,
                   41 / 840]
        self.B7 = [41 / 840, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 41 / 840, 0,
                   0]
        # stability polynomial of the 8th-order solution: G[m] = b8 A^(m-1) 1
        M = np.zeros((13, 13))
        for i, row in enumerate(A):
            M[i, :len(row)] = row
        v, self.G = np.ones(13), [1.0]
        for _ in range(12):
            self.G.append(float(np.dot(self.B8, v)))
            v = M @ v


class _Plain:
    """The generator in plain torch: states are real [n, 2B], the real parts
    of the B pulses and then their imaginary parts."""

    def __init__(self, case, seed):
        E, self.D = _system(case, seed)
        self.E = torch.as_tensor(np.concatenate(E), device="cuda")[:, None]
        self.n, self.B, self.length = _sizes(case), _batch(case), case["gauge"] == "l"
        if not self.length:
            self.upper = [-d for d in self.D]
        else:
            self.upper = self.D

    def load(self, x):
        t = torch.as_tensor(x.T, device="cuda")
        return torch.cat([t.real, t.imag], 1).contiguous()

    def store(self, x):
        t = x.detach()
        return torch.complex(t[:, :self.B], t[:, self.B:]).T.contiguous().cpu().numpy()

    def rhs(self, F, x):
        p = torch.split(x, self.n)
        W = []
        for L in range(len(self.n)):
            w = 0.0
            if L:
                w = w + self.D[L - 1].T @ p[L - 1]
            if L + 1 < len(self.n):
                w = w + self.upper[L] @ p[L + 1]
            W.append(w)
        W = torch.cat(W)
        B, re, im = self.B, x[:, :self.B], x[:, self.B:]
        if self.length:
            return torch.cat([self.E * im + F * W[:, B:], -self.E * re - F * W[:, :B]], 1)
        return torch.cat([self.E * im + F * W[:, :B], -self.E * re + F * W[:, B:]], 1)

    def step(self, G, F, dt, x):
        v = G[12] * x
        for m in range(11, -1, -1):
            v = dt * self.rhs(F, v) + G[m] * x
        return v

    def norm(self, x):
        return (x[:, :self.B] ** 2 + x[:, self.B:] ** 2).sum(0).sqrt()


def _fields(case, seed, t):
    """Field of every pulse at its time t[b]."""
    out = []
    for (I, w, cep, cycles), tb in zip(_pulses(case, seed), t):
        Eo = math.sqrt(I) / (1.0 if case["gauge"] == "l" else w)
        if case["shape"] == "sine":
            a = w / (2.0 * cycles)
            inside = 0.0 <= tb <= math.pi / a
            f = Eo * math.sin(a * tb) ** 2 * math.sin(w * tb + cep * 2 * math.pi / w)
        else:
            tau = cycles * 2.0 * math.pi / w
            fwhm = 2 + cycles // 10
            a = 0.5 * (2 * math.pi / w) * fwhm / 0.58870501125773734549
            inside = 0.0 <= tb <= tau
            f = Eo * math.exp(-((tb - 0.5 * tau) / a) ** 2) * math.sin(w * tb + cep)
        out.append(f if inside else 0.0)
    return out


def _kernel(K, T, t):
    """Weights [K] of the control samples at time t (Catmull-Rom)."""
    out = np.zeros(K)
    if not 0.0 <= t <= T:
        return out
    s = t / (T / (K - 1))
    k0 = min(int(math.floor(s)), K - 2)
    for k in range(k0 - 1, k0 + 3):
        d = abs(s - k)
        phi = 1 - 2.5 * d * d + 1.5 * d ** 3 if d <= 1 else \
            2 - 4 * d + 2.5 * d * d - 0.5 * d ** 3 if d < 2 else 0.0
        if 0 <= k < K:
            out[k] = phi
    return out


def exact(case, seed):
    tab, p = _Tableau(), _Plain(case, seed)
    x, op = p.load(_states(case, seed)[:p.B]), case["op"]
    if op in ("rhs", "step"):
        F = 0.03 + 0.01 * (seed % 7)
        v = p.rhs(F, x) if op == "rhs" else p.step(tab.G, F, case["dt"], x)
        return p.store(v)[0]
    t = _start_times(case, seed)
    if op == "adaptive":
        return _exact_adaptive(case, seed, tab, p, x, t)
    if op in ("grad", "bgrad"):
        return _exact_gradient(case, seed, tab, p, x, float(t[0]))
    dt, B = case["dt"], p.B
    steps = _step_counts(case) if op == "advance" else [case["steps"]]
    M = max(steps)
    pop, nrm, fld = np.full((B, M + 1), np.nan), np.full((B, M), np.nan), []
    pops, nrms = [x[0, :B] ** 2 + x[0, B:] ** 2], []
    last = torch.as_tensor(steps, device="cuda")
    t = list(t)
    for k in range(M):
        F = _fields(case, seed, [v + dt for v in t])
        t = [v + dt for v in t]
        fld.append(F[0])
        v = p.step(tab.G, torch.tensor(F, device="cuda", dtype=torch.float64), dt, x)
        norm = p.norm(v)
        v = v / torch.cat([norm, norm])
        on = (last > k).repeat(2)
        x = torch.where(on, v, x)
        nrms.append(norm)
        pops.append(x[0, :B] ** 2 + x[0, B:] ** 2)
    pops, nrms = torch.stack(pops, 1).cpu().numpy(), torch.stack(nrms, 1).cpu().numpy()
    for b in range(B):
        pop[b, :steps[b] + 1] = pops[b, :steps[b] + 1]
        nrm[b, :steps[b]] = nrms[b, :steps[b]]
    if op == "propagate":
        return p.store(x)[0], pop[0], np.array(fld), nrm[0]
    return p.store(x), pop, nrm


def _exact_adaptive(case, seed, tab, p, x, t):
    B, t_end = p.B, t + _windows(case, seed)
    t, h, done = t.copy(), np.full(B, 0.05), np.zeros(B, bool)
    while not done.all():
        rem = t_end - t
        last = h >= rem
        hatt = np.where(done, 0.0, np.where(last, rem, h))
        hd = torch.as_tensor(hatt, device="cuda")
        hc = torch.cat([hd, hd])
        K = []
        for s in range(13):
            F = _fields(case, seed, t + tab.C[s] * hatt)
            y = x
            for a, k in zip(tab.A[s], K):
                if a:
                    y = y + (hc * a) * k
            K.append(p.rhs(torch.tensor(F, device="cuda", dtype=torch.float64), y))
        new = x + sum((hc * b) * k for b, k in zip(tab.B8, K) if b)
        e = hc * (41 / 840) * (K[0] + K[10] - K[11] - K[12])
        mod = lambda v: (v[:, :B] ** 2 + v[:, B:] ** 2).sqrt()  # noqa: E731
        err = (mod(e) / (1e-10 + 1e-10 * torch.maximum(mod(x), mod(new)))).amax(0).cpu().numpy()
        ok = (err <= 1.0) & ~done
        fac = np.clip(0.9 * np.maximum(err, 1e-300) ** -0.125, 0.2, 5.0)
        on = torch.as_tensor(ok, device="cuda").repeat(2)
        norm = p.norm(new)
        x = torch.where(on, new / torch.cat([norm, norm]), x)
        t = np.where(ok, np.where(last, t_end, t + hatt), t)
        h = np.where(ok, np.minimum(hatt * fac, 0.15), np.where(done, h, hatt * np.minimum(fac, 1)))
        done |= ok & last
    return p.store(x), None, None, t


def _exact_gradient(case, seed, tab, p, x, t):
    dt, steps, B, T = case["dt"], case["steps"], p.B, (case["steps"] + 1) * case["dt"]
    u = torch.as_tensor(_controls(case, seed), device="cuda")
    W, F0 = [], []
    for _ in range(steps):
        F0.append(_fields(case, seed, [t + dt] * B))
        W.append(_kernel(case["controls"], T, t + dt))
        t += dt
    W = torch.as_tensor(np.array(W), device="cuda")
    F = (torch.tensor(F0, device="cuda", dtype=torch.float64).T + u @ W.T)
    # the state at every step, then one step at a time backwards
    xs = [x]
    with torch.no_grad():
        for k in range(steps):
            v = p.step(tab.G, F[:, k], dt, xs[-1])
            norm = p.norm(v)
            xs.append(v / torch.cat([norm, norm]))
    keep = (p.E >= 0).to(torch.float64)
    end = xs[-1]
    J = (keep * (end[:, :B] ** 2 + end[:, B:] ** 2)).sum(0)
    lam, dF = 2.0 * keep * end, torch.zeros(B, steps, device="cuda", dtype=torch.float64)
    for k in range(steps - 1, -1, -1):
        f, xk = F[:, k].clone().requires_grad_(), xs[k].clone().requires_grad_()
        v = p.step(tab.G, f, dt, xk)
        norm = p.norm(v)
        (v / torch.cat([norm, norm])).backward(lam)
        lam, dF[:, k] = xk.grad, f.grad
    J, g, dF = J.cpu().numpy(), (dF @ W).cpu().numpy(), dF.cpu().numpy()
    if case["op"] == "grad":
        return float(J[0]), g[0], dF[0]
    return J, g, dF
