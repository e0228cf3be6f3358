"""Cases for measuring the framework: what a program that uses it has it do, over the sizes it is used at.

A program builds a mechanism once (its tables on the GPU, the transport fits for its normalisation) and then
calls the per-cell evaluations over and over, from one state (an ODE solver's right-hand side, a boundary
condition) to the millions of cells of a flow field; it trains a transport surrogate and evaluates it, and
integrates batches of reactors. Mechanisms, cell distributions and shapes are the repository's own seeded
workloads (combustion_gb300/synthetic.py): 10 species / 25 reactions, 53 / 325 and 250 / 1,500.
"""
import functools
import math

import numpy as np
import torch

import combustion_gb300 as cb
from combustion_gb300 import reactors as RX
from combustion_gb300 import surrogate as SUR
from combustion_gb300 import synthetic

F64 = torch.float64


def listed():
    return [
        # One state of the 53-species mechanism at one pressure: the call an ODE solver or a boundary condition
        # makes, where only latency counts.
        {"name": "rates_k53_one_state", "kind": "rates", "config": "k53", "n": 1, "uniform": True},
        # The small mechanism on 65,536 cells (rates and transport of a 256 x 256 field).
        {"name": "fused_k10_65536", "kind": "fused", "config": "k10", "n": 65536},
        # A 100 x 100 field and a ragged row: an ordinary small field, less than one cell per resident thread.
        {"name": "rates_k53_10100", "kind": "rates", "config": "k53", "n": 10100, "uniform": True},
        # Transport alone on a 2-D field (properties are often refreshed less often than the rates), odd size.
        {"name": "transport_k53_90301", "kind": "transport", "config": "k53", "n": 90301},
        # The rate of progress of every reaction (reaction path analysis) on a 2-D field.
        {"name": "reaction_rates_k53_131072", "kind": "reaction_rates", "config": "k53", "n": 131072},
        # The full evaluation of a 3-D field: rates and transport of 2^22 cells, per-cell pressure.
        {"name": "fused_k53_4194304", "kind": "fused", "config": "k53", "n": 1 << 22},
        # The same call on host arrays (a solver that keeps its field on the host), copies included.
        {"name": "fused_host_k53_262144", "kind": "fused_host", "config": "k53", "n": 262144},
        # The large mechanism, a 2-D field.
        {"name": "fused_k250_32768", "kind": "fused", "config": "k250", "n": 32768},
        # The mixed-precision form on a 3-D field of odd size.
        {"name": "fused_mixed_k53_1000003", "kind": "fused_mixed", "config": "k53", "n": 1000003},
        # The learned transport surrogate with its trust gate and audit on a 3-D field.
        {"name": "surrogate_k53_524288", "kind": "surrogate", "config": "k53", "n": 524288},
        # Training the surrogate's network: 32 steps of 65,536 rows, width 256, 4 hidden layers.
        {"name": "train_k53_32x65536", "kind": "train", "config": "k53", "n": 65536, "steps": 32},
        # A batch of reactors to 1 ms with the default options.
        {"name": "reactors_k53_512", "kind": "reactors", "config": "k53", "n": 512},
    ]


# Most cells of a drawn case per kind and mechanism: none costs more than the 2^22-cell evaluation.
_MOST = {
    "rates": {"k10": 1 << 22, "k53": 1 << 22, "k250": 1 << 18},
    "transport": {"k10": 1 << 22, "k53": 1 << 22, "k250": 1 << 17},
    "fused": {"k10": 1 << 22, "k53": 1 << 22, "k250": 1 << 17},
    "reaction_rates": {"k10": 1 << 21, "k53": 1 << 20, "k250": 1 << 16},
    "fused_host": {"k10": 1 << 20, "k53": 1 << 20},
    "rates_mixed": {"k10": 1 << 22, "k53": 1 << 22, "k250": 1 << 18},
    "fused_mixed": {"k10": 1 << 22, "k53": 1 << 22, "k250": 1 << 18},
    "surrogate": {"k10": 1 << 21, "k53": 1 << 21},
    "reactors": {"k10": 512, "k53": 512},
}
_LEAST = {"surrogate": 4096, "reactors": 32}


def draw(rng):
    kind = rng.choice(["rates", "rates", "transport", "transport", "fused", "fused", "reaction_rates", "fused_host",
                       "rates_mixed", "fused_mixed", "surrogate", "train", "reactors"])
    if kind == "train":
        return {"kind": kind, "config": rng.choice(["k10", "k53"]), "n": 128 * rng.randint(32, 512),
                "steps": rng.randint(8, 40)}
    config = rng.choice([c for c in ("k10", "k53", "k53", "k250") if c in _MOST[kind]])
    lo, hi = math.log(_LEAST.get(kind, 1)), math.log(_MOST[kind][config])
    n = int(round(math.exp(lo + (hi - lo) * rng.random())))
    case = {"kind": kind, "config": config, "n": max(1, n | 1 if rng.random() < 0.5 else n)}
    case["n"] = min(case["n"], _MOST[kind][config])
    if kind in ("rates", "rates_mixed") and rng.random() < 0.3:
        case["uniform"] = True
    return case


# ---- what a program keeps: mechanisms with their transport fits, trained networks --------------------------
@functools.lru_cache(maxsize=None)
def _data(config, reactor=False):
    return synthetic.generate_reactor_mechanism(config) if reactor else synthetic.generate_mechanism(config)


@functools.lru_cache(maxsize=None)
def _mechanism(config, reactor=False):
    m = _data(config, reactor)
    h = cb.Mechanism(m)
    h.transport_setup(*synthetic.transport_scales(m))
    return h


@functools.lru_cache(maxsize=None)
def _trained(config):
    """A network of the default shape after a short training (its accuracy does not change what a call costs)."""
    s = SUR.Surrogate(_mechanism(config), width=256, hidden_layers=4, batch=16384, lr_final=1e-5, seed=3)
    s.generate(1 << 18, SUR.distribution(config, seed=2))
    s.train(300)
    return s


def _cells(case, seed):
    """Cells of the configuration's distribution in the rates layout [K+3, n], on the GPU."""
    c = SUR.generate_cells(_mechanism(case["config"]), case["n"], SUR.distribution(case["config"], seed=100 + seed))
    if case.get("uniform"):  # every cell at the first cell's pressure (V adjusted to keep the ideal-gas total)
        c[3] *= c[0] / c[0, 0]
        c[0], c[1] = c[0, 0].clone(), c[1, 0].clone()
    return c


def _transport_inputs(config, c):
    """The transport call's inputs (sum n, T/T0, n_0 ..) of rates-layout cells."""
    T0 = synthetic.transport_scales(_data(config))[0]
    return torch.cat([(c[0] * c[3] / c[2])[None], (c[2] / T0)[None], c[4:]]).contiguous()


def prepare(case, seed):
    kind, config, n = case["kind"], case["config"], case["n"]
    s = {"case": case}
    if kind == "reactors":
        mech = _mechanism(config, True)
        s["reactors"] = RX.Reactors(mech, n)
        s["initial"] = RX.initial_states(mech.K, n, seed=400 + seed)
        s["reactors"].set_state(*s["initial"])
        s["reactors"].autotune()
        return s
    mech = _mechanism(config)
    K, A, R = mech.K, mech.A, mech.R
    if kind == "train":
        s["network"] = SUR.Surrogate(mech, width=256, hidden_layers=4, batch=n, lr_final=1e-5, seed=30 + seed)
        s["network"].generate(2 * n, SUR.distribution(config, seed=200 + seed))
        return s
    s["mech"], cells = mech, _cells(case, seed)
    if kind == "transport":
        s["in"] = _transport_inputs(config, cells)
    elif kind == "reaction_rates":
        s["in"] = torch.cat([cells[:1], cells[2:]]).contiguous()
    else:
        s["in"] = cells
    empty = (lambda rows: torch.empty((rows, n), dtype=F64, pin_memory=True).numpy()) if kind == "fused_host" else (
        lambda rows: torch.empty((rows, n), dtype=F64, device="cuda"))
    if kind == "fused_host":
        host = torch.empty(cells.shape, dtype=F64, pin_memory=True)
        host.copy_(cells)
        s["in"] = host.numpy()
    if kind in ("rates", "fused", "fused_host", "rates_mixed", "fused_mixed"):
        s["rates"] = empty(A + 2)
    if kind in ("transport", "fused", "fused_host", "fused_mixed", "surrogate"):
        s["transport"] = empty(K + 2)
    if kind == "reaction_rates":
        s["progress"] = empty(R)
    if kind == "surrogate":
        s["network"] = _trained(config)
    return s


def run(s):
    case = s["case"]
    kind, uniform = case["kind"], bool(case.get("uniform"))
    if kind in ("rates", "rates_mixed"):
        return s["mech"].rates(s["in"], s["rates"], uniform_pressure=uniform, mixed=kind == "rates_mixed")
    if kind == "transport":
        return s["mech"].transport(s["in"], s["transport"])
    if kind == "reaction_rates":
        return s["mech"].reaction_rates(s["in"], s["progress"])
    if kind in ("fused", "fused_host", "fused_mixed"):
        return s["mech"].rates_transport(s["in"], s["rates"], s["transport"], mixed=kind == "fused_mixed")
    if kind == "surrogate":
        stats = s["network"].transport(s["in"], s["transport"])
        return {"transport": s["transport"], "fallback": stats["fallback_cells"], "audited": stats["audited_cells"]}
    if kind == "train":
        losses = s["network"].train(case["steps"])
        return {"losses": losses, "params": s["network"].params()}
    r = s["reactors"]
    r.set_state(*s["initial"])
    r.integrate()
    got = r.results()
    return {"ignition_delay": got["ignition_delay"], "state": got["state"], "status": got["status"]}


# ---- the work that a pass cannot do without ------------------------------------------------------------------
def _cell_flops(config):
    """(rates, transport) operations per cell: multiply-adds as 2, an exponential, logarithm, division or square
    root as 1."""
    r, t = _mechanism(config).work_model()
    count = lambda w: w["flops"] + w["exps"] + w["logs"] + w["divs"] + w["sqrts"]  # noqa: E731
    return count(r), count(t)


def work(case):
    kind, config, n = case["kind"], case["config"], case["n"]
    m = _data(config, kind == "reactors")
    K, A, R = m.K, m.K - 1, m.R
    if kind == "reactors":  # at least a few hundred steps, each a right-hand side and a triangular solve per iteration
        rates, _ = _cell_flops(config)
        N = A + 2
        return {"bytes": 8.0 * n * (2 * N + 2), "flops": 400.0 * n * (2.4 * rates + 2 * 2.0 * N * N)}
    if kind in ("surrogate", "train"):
        wide = 64 * math.ceil((K + 2) / 64)
        weights = 2 * wide * 256 + 3 * 256 * 256
        if kind == "surrogate":
            return {"bytes": 8.0 * n * (K + 3 + K + 2), "flops": 2.0 * weights * n}
        per_step = 2.0 * n * wide + 4.0 * n * wide + 4 * 4.0 * weights
        return {"bytes": per_step * case["steps"], "flops": 6.0 * weights * n * case["steps"]}
    rates, transport = _cell_flops(config)
    ins = K + 1 if case.get("uniform") or kind == "transport" else K + 2 if kind == "reaction_rates" else K + 3
    outs = {"rates": A + 2, "rates_mixed": A + 2, "transport": K + 2, "reaction_rates": R}.get(kind, A + K + 4)
    flops = {"rates": rates, "rates_mixed": rates, "transport": transport, "reaction_rates": rates}.get(
        kind, rates + transport)
    return {"bytes": 8.0 * n * (ins + outs), "flops": flops * n}


# ---- the same values in 64 bits, plain torch -----------------------------------------------------------------
_R_GAS = 1.380649e-23 * 6.02214076e23
_F32_MAX, _F32_TINY = float(np.finfo(np.float32).max), float(np.finfo(np.float32).tiny)


def _polynomial(a, T, split, terms):
    """Per-species piecewise polynomials: sum_i terms[i](a) * power_i(T), the piece chosen by T <= split."""
    v = [sum(c * p for c, p in terms(a[piece])) for piece in (0, 1)]
    return v[0] if math.isnan(split) else torch.where(T <= split, v[0], v[1])


def _progress(m, P_R, T, C):
    """Rate of progress of every reaction, one after the other: (reaction, its tensor over the cells)."""
    K, R = m.K, m.R
    lnT, rT = torch.log(T), 1.0 / T
    Ctot = P_R * rT
    cap = np.float32(np.cbrt(_F32_MAX))  # of e^-g; that of e^g is the largest whose cube stays finite in 32 bits
    largest = cap
    with np.errstate(over="ignore"):
        while np.isinf(np.float32(largest * largest) * largest):
            largest = np.nextafter(largest, np.float32(0))
    cap, largest = float(cap), float(largest)
    gibbs = []
    for k in range(K - 1):
        gibbs.append(_polynomial(m.nasa7[k], T, m.nasa7_split[k], lambda a: [
            (a[0] - a[6], 1.0), (-a[0], lnT), (-a[1] / 2, T), (-a[2] / 6, T ** 2), (-a[3] / 12, T ** 3),
            (-a[4] / 20, T ** 4), (a[5], rT)]))

    def arrhenius(A, b, Ea):
        return torch.clamp(torch.exp(math.log(A) + b * lnT - Ea * rT), max=_F32_MAX)

    for r in range(R):
        model = int(m.model[r])
        A, b, Ea = (float(v) for v in m.rate[r])
        k = arrhenius(A, b, Ea) if model != synthetic.TROE else None
        if model in (synthetic.THREE_BODY, synthetic.TROE):
            M = Ctot.clone()
            for j in np.flatnonzero(m.efficiencies[r] != 1.0):
                M += (m.efficiencies[r, j] - 1.0) * C[j]
        if model == synthetic.THREE_BODY:
            k = k * M
        elif model == synthetic.TROE:
            A0, b0, Ea0 = (float(v) for v in m.k0[r])
            ki = arrhenius(1.0, b, Ea)
            Pr = M * arrhenius(A0 / A, b0, Ea0) / (ki + _F32_TINY)
            a, T3, T1, T2 = (float(v) for v in m.troe[r])
            F = (1.0 - a) * torch.exp(-T / T3) + a * torch.exp(-T / T1)
            if math.isfinite(T2):
                F = F + torch.exp(-T2 * rT)
            lnF = torch.log(F)
            x = torch.log(Pr + _F32_TINY) - 0.67 * lnF - 0.4 * math.log(10.0)
            f1 = x / (-0.14 * x - 1.27 * lnF + 0.75 * math.log(10.0))
            k = torch.exp(lnF / (f1 * f1 + 1.0)) * (A * ki) * Pr / (Pr + 1.0)
        elif model != synthetic.ELEMENTARY:
            raise ValueError("the seeded mechanisms have no reaction of this model")
        forward, backward, kc = 1.0, 1.0, 1.0
        for j in np.flatnonzero(m.reactants[r]):
            forward = forward * C[j] ** int(m.reactants[r, j])
        for j in np.flatnonzero(m.products[r]):
            backward = backward * C[j] ** int(m.products[r, j])
        net = m.products[r].astype(int) - m.reactants[r].astype(int)
        for j in np.flatnonzero(net):
            e = torch.clamp(torch.exp(gibbs[j]), max=largest) if net[j] > 0 else torch.clamp(
                torch.exp(-gibbs[j]), max=cap)
            kc = kc * e ** int(abs(net[j]))
        kc = kc * (101325.0 / _R_GAS * rT) ** int(-net.sum())
        yield r, k * (forward - kc * backward)


def _concentrations(P_R, T, V, n):
    C = torch.clamp(n, min=0.0) / V
    return torch.cat([C, (P_R / T - C.sum(0))[None]])


def _rates_exact(m, P_R, rP, T, V, n):
    C = _concentrations(P_R, T, V, n)
    A = m.K - 1
    out = torch.zeros((A + 2, T.numel()), dtype=F64, device=T.device)
    w = out[2:]
    for r, q in _progress(m, P_R, T, C):
        net = m.products[r].astype(int) - m.reactants[r].astype(int)
        for j in np.flatnonzero(net):
            w[j] += float(net[j]) * q
    E, Cp, dE = torch.zeros_like(T), torch.zeros_like(T), torch.zeros_like(T)
    for k in range(m.K):
        cp = _polynomial(m.nasa7[k], T, m.nasa7_split[k], lambda a: [(a[i], T ** i) for i in range(5)])
        Cp += cp * C[k]
        if k < A:
            h = _polynomial(m.nasa7[k], T, m.nasa7_split[k], lambda a: [
                (a[0], 1.0), (a[1] / 2, T), (a[2] / 3, T ** 2), (a[3] / 4, T ** 3), (a[4] / 5, T ** 4), (a[5], 1.0 / T)])
            E += w[k] * h
            dE += (1.0 - m.molar_mass[k] / m.molar_mass[-1]) * w[k]
    d = -E / Cp
    out[0] = T * d
    out[1] = V * (d + rP * T * dE)
    return out


def _transport_exact(config, N, Tn, n):
    """lambda/lambda0, mu/mu0 and rho D_k/mu0 from the mechanism's fitted polynomials (its parameters)."""
    m = _data(config)
    T0, mu0, l0 = synthetic.transport_scales(m)
    cond, visc, diff = (torch.from_numpy(v).to(Tn.device) for v in _mechanism(config).transport_coefficients())
    K, W = m.K, torch.from_numpy(m.molar_mass).to(Tn.device)
    cond, visc = cond * (math.sqrt(T0) / (2 * l0)), visc * (math.sqrt(math.sqrt(T0)) / math.sqrt(mu0))
    diff = diff.reshape(K, K, 5) * (math.sqrt(T0) / (_R_GAS * mu0))
    L = torch.stack([torch.log(Tn) ** i for i in range(5)])
    X = torch.cat([n, (N - n.sum(0))[None]])
    VT = torch.sqrt(Tn)
    MN = (W[:, None] * X).sum(0)
    c, v = cond @ L, visc @ L
    out = torch.empty((K + 2, Tn.numel()), dtype=F64, device=Tn.device)
    out[0] = ((X * c).sum(0) / N + N / (X / c).sum(0)) * VT
    mu, S = torch.zeros_like(Tn), torch.zeros_like(X)
    for k in range(K):
        va = torch.sqrt(1.0 / math.sqrt(8.0) / torch.sqrt(1.0 + W[k] / W))
        b = va * (W / W[k]) ** 0.25
        mu += X[k] * v[k] ** 2 / (X * (va[:, None] + b[:, None] * v[k] / v) ** 2).sum(0)
        if k:
            r = 1.0 / (diff[k, :k] @ L)
            S[k] += (X[:k] * r).sum(0)
            S[:k] += X[k] * r
    out[1] = VT * mu
    for k in range(K):
        out[2 + k] = (MN * VT - VT * W[k] * X[k]) / S[k]
    return out


def _by_chunks(n, rows, fn):
    """fn(lo, hi) over chunks small enough for the temporaries."""
    step = max(1, (1 << 25) // rows)
    return torch.cat([fn(lo, min(n, lo + step)) for lo in range(0, n, step)], dim=1)


def _exact_rates(case, c):
    m = _data(case["config"])
    return _by_chunks(case["n"], m.K, lambda a, b: _rates_exact(m, c[0, a:b], c[1, a:b], c[2, a:b], c[3, a:b], c[4:, a:b]))


def _exact_transport(config, c):
    T0 = synthetic.transport_scales(_data(config))[0]
    return _by_chunks(c.shape[1], c.shape[0], lambda a, b: _transport_exact(
        config, c[0, a:b] * c[3, a:b] / c[2, a:b], c[2, a:b] / T0, c[4:, a:b]))


def _features(config, c, norm):
    """The surrogate's raw inputs log(T/T0), log(P/atm), X_0 .. X_{K-1}, and the same normalised."""
    T0 = synthetic.transport_scales(_data(config))[0]
    N = c[0] * c[3] / c[2]
    raw = torch.cat([torch.log(c[2] / T0)[None], torch.log(c[0] * (_R_GAS / 101325.0))[None], c[4:] / N,
                     ((N - c[4:].sum(0)) / N)[None]])
    mean, rstd = (torch.from_numpy(norm[k]).double().to(c.device)[:, None] for k in ("in_mean", "in_rstd"))
    return raw, (raw - mean) * rstd


def _forward(layers, x):
    for i, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if i + 1 < len(layers):
            x = torch.nn.functional.silu(x)
    return x


def _exact_train(case, seed):
    s = prepare(case, seed)["network"]
    config, n, steps, K = case["config"], case["n"], case["steps"], _data(case["config"]).K
    c = SUR.generate_cells(_mechanism(config), 2 * n, SUR.distribution(config, seed=200 + seed))
    norm = s.normalisation()
    x = _features(config, c, norm)[1].T
    out_mean, out_std = (torch.from_numpy(norm[k]).double().cuda() for k in ("out_mean", "out_std"))
    y = ((torch.log(_exact_transport(config, c)).T) - out_mean) / out_std
    x, y = (torch.nn.functional.pad(v, (0, s.info.n_in - K - 2)) for v in (x, y))
    p = torch.from_numpy(s.params()).double().cuda().requires_grad_()
    m1, m2, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for t in range(1, steps + 1):
        lo = ((t - 1) % 2) * n
        loss = ((_forward(s.layers(p), x[lo:lo + n]) - y[lo:lo + n])[:, :K + 2] ** 2).mean()
        (g,) = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        with torch.no_grad():
            lr = 1e-5 + 0.5 * (1e-3 - 1e-5) * (1.0 + math.cos(math.pi * (t - 1) / max(1, steps - 1)))
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            p = p - lr * (m1 / (1 - 0.9 ** t)) / (torch.sqrt(m2 / (1 - 0.999 ** t)) + 1e-8)
        p.requires_grad_()
    return {"losses": np.array(losses), "params": p.detach()}


def exact(case, seed):
    kind, config, n = case["kind"], case["config"], case["n"]
    if kind == "reactors":  # an integration to tighter tolerances takes minutes
        return None
    if kind == "train":
        return _exact_train(case, seed)
    m, c = _data(config), _cells(case, seed)
    if kind in ("rates", "rates_mixed"):
        return _exact_rates(case, c)
    if kind == "transport":
        t = _transport_inputs(config, c)
        return _by_chunks(n, m.K, lambda a, b: _transport_exact(config, t[0, a:b], t[1, a:b], t[2:, a:b]))
    if kind == "reaction_rates":
        def progress(a, b):
            q = torch.empty((m.R, b - a), dtype=F64, device=c.device)
            for r, v in _progress(m, c[0, a:b], c[2, a:b], _concentrations(c[0, a:b], c[2, a:b], c[3, a:b], c[4:, a:b])):
                q[r] = v
            return q
        return _by_chunks(n, m.R, progress)
    if kind in ("fused", "fused_host", "fused_mixed"):
        return _exact_rates(case, c), _exact_transport(config, c)
    s = _trained(config)  # the surrogate: its network in 64 bits, cells outside its range and audited ones exactly
    norm = s.normalisation()
    layers = s.layers(torch.from_numpy(s.params()).double().cuda())
    lo, hi, mean, std = (torch.from_numpy(norm[k]).double().cuda() for k in ("in_lo", "in_hi", "out_mean", "out_std"))

    def network(a, b):
        raw, x = _features(config, c[:, a:b], norm)
        x = torch.nn.functional.pad(x.T, (0, s.info.n_in - m.K - 2))
        y = torch.exp(_forward(layers, x)[:, :m.K + 2] * std + mean).T
        f = raw.float().double()
        own = ((f < lo[:, None]) | (f > hi[:, None])).any(0)
        own |= torch.arange(a, b, device=c.device) % 1024 == 7919 % 1024
        y[:, own] = _exact_transport(config, c[:, a:b][:, own]) if bool(own.any()) else y[:, own]
        return y
    return {"transport": _by_chunks(n, 1024, network), "fallback": None, "audited": None}
