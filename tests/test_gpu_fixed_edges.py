"""Calls at the edges of the plain fixed-point form: states it must leave to the FP64 form, words at the ends of their
range, threads and outputs that share what a call uses.

Where a cell has to take the FP64 form, its outputs are compared with the same mechanism plus one reaction that changes
nothing (a species reacting to itself) and whose constants no fixed-point word holds: all of its cells take that form.
"""
import copy

import numpy as np
import pytest

import util
from combustion_gb300 import synthetic

pytestmark = pytest.mark.gpu


def dev(x):
    import torch
    return torch.tensor(np.array(x), dtype=torch.float64, device="cuda")


def with_fp64_form(m):
    """m with one more reaction, S0 -> S0 at exp(-2e5 K / T): the rates' values stay, their form is the FP64 one."""
    m = copy.deepcopy(m)
    one = np.zeros((1, m.K), dtype=np.uint8)
    one[0, 0] = 1
    m.reactants, m.products = np.vstack([m.reactants, one]), np.vstack([m.products, one])
    m.model = np.append(m.model, np.int32(synthetic.IRREVERSIBLE))
    for name, row in (("rate", (1.0, 0.0, 2e5)), ("k0", 0.0), ("troe", 0.0), ("sri", 0.0), ("efficiencies", 1.0)):
        a = getattr(m, name)
        setattr(m, name, np.vstack([a, np.full((1, a.shape[1]), row)]))
    return m


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
def test_states_of_the_fp64_form(config):
    """Non-finite and non-positive states give what the FP64 form gives, NaN and infinity by NaN and infinity: in calls
    of one cell per block, per warp and per thread."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech, ref, o = cb.Mechanism(m), cb.Mechanism(with_fp64_form(m)), oracle.Oracle(m)
    n, K = 48, m.K
    cells = synthetic.generate_cells(K, n, config, seed=37)
    pin = np.array(o.reaction_rates_inputs(cells))  # P/R, T, V, n_0 ..
    states = []  # (row, value); rows 0 .. 2 are P/R, T, V
    for k in (0, K // 2, K - 2):
        states += [(3 + k, np.nan), (3 + k, np.inf), (3 + k, -np.inf), (3 + k, -1.0)]
    states += [(2, np.nan), (2, 0.0), (2, -1.0), (2, -1e-6), (2, np.inf), (2, 1e-305), (0, np.nan), (0, 0.0), (0, -100.0),
               (0, np.inf), (1, np.nan), (1, -300.0), (1, 0.0), (1, np.inf)]
    for c, (row, value) in enumerate(states):
        pin[row, c] = value
    pin[3:, len(states)] = 0.0
    with np.errstate(divide="ignore"):
        rin = np.vstack([pin[:1], 1.0 / pin[:1], pin[1:]])
    with np.errstate(all="ignore"):
        scales = o.rates(list(rin), scale=True)[1], o.reaction_rates(list(pin), scale=True)[1]
    reps = {"k10": 64, "k53": 400, "k250": 400}[config] * 152 // n + 1
    for name, x, sc, rows in (("rates", rin, scales[0], m.active() + 2), ("reaction_rates", pin, scales[1], m.R)):
        for r in (1, 40, reps):
            got = []
            for h in (mech, ref):
                # one output row per reaction of its own mechanism
                t = torch.full((rows + (name == "reaction_rates" and h is ref), n * r), 7.0, dtype=torch.float64, device="cuda")
                getattr(h, name)(dev(np.tile(x, (1, r))), t)
                h.synchronize()
                got.append(t[:rows, -n:].cpu().numpy())
            a, b = got
            for c in range(len(states) + 1):
                what = f"{name}, {n * r} cells, state {states[c] if c < len(states) else 'no amounts'}"
                assert np.array_equal(np.isnan(a[:, c]), np.isnan(b[:, c])), what
                assert np.array_equal(np.isinf(a[:, c]) * np.sign(a[:, c]), np.isinf(b[:, c]) * np.sign(b[:, c]),
                                      equal_nan=True), what
            both = np.isfinite(a) & np.isfinite(sc)
            assert (util.cond_err(a, b, sc)[both] <= util.PLAIN_TOL).all()


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("mixed", [False, True])
def test_fused_call_with_rates_over_the_cells(config, mixed):
    """A fused call whose species rates overwrite the cells' amounts: the transport is of the overwritten cells, as in two
    calls one after the other, at sizes where the two kernels otherwise run beside each other."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech = cb.Mechanism(m)
    mech.transport_setup(*synthetic.transport_scales(m))
    assert m.active() == m.K - 1
    for n in {"k10": (1, 300, 5000, 70001), "k53": (1, 300, 10100, 70001), "k250": (1, 456, 12001)}[config]:
        x = dev(oracle.Oracle(m).rates_inputs(synthetic.generate_cells(m.K, n, config, seed=7)))
        got = []
        for fused in (True, False):
            y, d = x.clone(), torch.empty((2, n), dtype=torch.float64, device="cuda")
            r = list(d) + list(y[4:])
            t = torch.full((m.K + 2, n), 7.0, dtype=torch.float64, device="cuda")
            if fused:
                mech.rates_transport(y, r, t, mixed=mixed)
            else:
                mech.rates(y, r, mixed=mixed)
                mech.rates_transport(y, torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda"), t, mixed=mixed)
            mech.synchronize()
            got.append(torch.cat([y, d, t]).nan_to_num(-3.0))
        assert torch.equal(*got)


def _words(v, low):
    """v = hi 2^low + lo, lo balanced, of Python integers."""
    hi = (v + (1 << (low - 1))) >> low
    return hi, v - (hi << low)


@pytest.mark.parametrize("power", [11, 13])
@pytest.mark.parametrize("kind", ["gibbs", "enthalpy", "heat-capacity"])
def test_low_words_at_their_end(kind, power):
    """Polynomials whose coefficients' low words are all close to -2^28, just below the end of a piece's temperatures (T /
    2^11 or T / 2^13 close to 1): the sum of their cross products is then as large as any mechanism's."""
    import torch
    import combustion_gb300 as cb
    import oracle
    LD = np.longdouble
    m = copy.deepcopy(util.mechanism("k10"))
    T = 2.0 ** power * (1.0 - 2.0 ** -31)
    L = 29
    target = -(1 << 28) + 256
    log2e = 1 / np.log(LD(2))
    # (coefficient index, factor to the polynomial's own, bits below the binary point of its two words, power of T)
    poly = {"gibbs": [(0, -1.0, 53, 0), (5, log2e, 43, -1), (1, -log2e / 2, 47, 1), (2, -log2e / 6, 47, 2),
                      (3, -log2e / 12, 47, 3), (4, -log2e / 20, 47, 4)],
            "enthalpy": [(5, 1.0, 43, -1), (1, 0.5, 47, 1), (2, LD(1) / 3, 47, 2), (3, 0.25, 47, 3), (4, LD(1) / 5, 47, 4)],
            "heat-capacity": [(1, 1.0, 47, 1), (2, 1.0, 47, 2), (3, 1.0, 47, 3), (4, 1.0, 47, 4)]}[kind]
    largest = 0
    for k in range(m.K):
        a2 = b2 = 0
        for i, factor, bits, n in poly:
            scale = LD(factor) * LD(2) ** (power * max(n, 0) + bits)
            hi, _ = _words(int(np.rint(LD(m.nasa7[k, 1, i]) * scale)), L)
            m.nasa7[k, 1, i] = float((LD(hi) * 2 ** L + target) / scale)
            w = _words(int(np.rint(LD(m.nasa7[k, 1, i]) * scale)), L)
            t = {0: np.log2(LD(T)) * LD(2) ** 56, -1: LD(2) ** 66 / LD(T)}.get(n, LD(2.0 ** -power * T) ** n * LD(2) ** 59)
            t = _words(int(np.rint(t)), L)
            term = w[0] * t[1] + w[1] * t[0]
            if n > 0:
                b2 += term
            else:
                a2 += term
        largest = max(largest, abs(a2 + 8 * b2))
    assert largest > 1 << 63  # (what a 64-bit sum in units of the smaller words does not hold)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    cells = synthetic.generate_cells(m.K, 64, "k10", seed=41)
    cells.amounts *= cells.temperature / T
    cells.temperature[:] = T
    rin = o.rates_inputs(cells)
    out = torch.empty((mech.A + 2, cells.n), dtype=torch.float64, device="cuda")
    mech.rates(dev(rin), out)
    mech.synchronize()
    ref, sc = o.rates(rin, scale=True)
    e = util.cond_err(out.cpu().numpy(), ref, sc)
    print(f"{kind}, T / 2^{power}: max cond err {e.max():.2e}")
    assert e.max() <= util.PLAIN_TOL


def test_calls_of_two_threads():
    """Two host threads, each with a handle and a stream of its own, whose calls take different amounts of shared memory
    from the same kernels (16 and 2 cells per block of one per warp; 8 warps per cell): every launch is accepted and
    every call gives what it gives alone."""
    import threading
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism("k10")
    x = dev(oracle.Oracle(m).rates_inputs(synthetic.generate_cells(m.K, 4000, "k10", seed=3)))
    errors = []

    def new(mech, n):
        return (torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda"),
                torch.empty((mech.K + 2, n), dtype=torch.float64, device="cuda"))

    def work(sizes, gate):
        try:
            mech, stream = cb.Mechanism(m), torch.cuda.Stream()
            mech.transport_setup(*synthetic.transport_scales(m))
            cells, outs = [x[:, :n].contiguous() for n in sizes], [new(mech, n) for n in sizes]
            alone = [new(mech, n) for n in sizes]
            for c, o in zip(cells, alone):
                mech.rates_transport(c, *o)
            torch.cuda.synchronize()
            gate.wait()
            for _ in range(1500):
                for c, (r, t) in zip(cells, outs):
                    mech.rates_transport(c, r, t, stream=stream)
                    mech.rates(c, r, stream=stream, mixed=True)
                    mech.rates(c, r, stream=stream)
            mech.synchronize(stream.cuda_stream)
            assert all(torch.equal(a, b) for p, q in zip(outs, alone) for a, b in zip(p, q))
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))
            gate.abort()

    gate = threading.Barrier(2)
    threads = [threading.Thread(target=work, args=(sizes, gate)) for sizes in ((2400, 1), (200, 400))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_large_call_after_small_ones():
    """A large call is as fast after a small call of another mechanism of the same capacity as before it (the split of
    shared memory and L1 that a small call prefers ends with it)."""
    import torch
    import combustion_gb300 as cb
    from combustion_gb300 import surrogate as S
    m = util.mechanism("k53")
    small = copy.deepcopy(m)  # the same species with a sixth of the reactions: smaller tables
    keep = np.arange(0, m.R) < m.K - 1  # (the generator's first K - 1 reactions change every species but the last)
    for name in ("reactants", "products", "model", "rate", "k0", "troe", "sri", "efficiencies"):
        setattr(small, name, getattr(m, name)[keep])
    mech, other = cb.Mechanism(m), cb.Mechanism(small)
    n = 1 << 20
    x = S.generate_cells(mech, n, S.distribution("k53", seed=5))
    out = torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda")

    def timed(mixed):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            mech.rates(x, out, mixed=mixed)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times))

    for mixed in (True, False):
        before = timed(mixed)
        other.rates(x[:, :50000], out[:, :50000], mixed=mixed)
        after = timed(mixed)
        print(f"mixed {mixed}: {before:.2f} ms, after a small call {after:.2f} ms")
        assert after < 1.1 * before


def concentrations(m, cells):
    """Ctot, S = 2^ex above it and every sum, and C of unit volumes, as every form computes them."""
    Ctot = cells.pressure_R * (1.0 / cells.temperature)
    total = np.zeros(cells.n)
    for k in range(m.K - 1):
        total = total + cells.amounts[k]
    return Ctot, np.frexp(np.maximum(total, Ctot))[1], np.vstack([cells.amounts, Ctot - total])


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("largest", [12.0, 17.0, 61.0, 128.5])
def test_third_body_sums(config, largest):
    """Third-body concentrations against long double, one species far more efficient than the others: the error is that
    of the words (sums in fixed point) and two roundings, below that of a chain of FP64 FMAs."""
    import torch
    import combustion_gb300 as cb
    LD = np.longdouble
    m = copy.deepcopy(util.mechanism(config))
    K, (s, p) = m.K, (0, 1)
    rows = np.flatnonzero(m.model == synthetic.THREE_BODY)
    rng = np.random.default_rng(5)
    for i, r in enumerate(rows):  # 1 M C_s, and nothing back where species p is absent
        m.reactants[r], m.products[r], m.rate[r] = 0, 0, (1.0, 0.0, 0.0)
        m.reactants[r, s] = m.products[r, p] = 1
        m.efficiencies[r] = rng.uniform(0.5, 3.0, K)
        m.efficiencies[r, 2 + i % (K - 2)] = largest
    assert m.active() == K - 1
    mech = cb.Mechanism(m)
    cells = synthetic.generate_cells(K, 512, config, seed=43)
    cells.amounts[p] = 0.0
    Ctot, ex, C = concentrations(m, cells)
    x = np.vstack([cells.pressure_R, cells.temperature, cells.volume, cells.amounts])
    out = torch.empty((m.R, cells.n), dtype=torch.float64, device="cuda")
    mech.reaction_rates(dev(x), out)
    mech.synchronize()
    out = out.cpu().numpy()
    worst = ratio = 0.0
    third = np.concatenate([np.flatnonzero(m.model == k) for k in (synthetic.THREE_BODY, synthetic.TROE)])  # (no Lindemann)
    for i, r in enumerate(rows):
        e = m.efficiencies[r].astype(LD) - 1
        M = Ctot + (e[:, None] * C).sum(0)
        four = np.abs(m.efficiencies[third[i // 4 * 4:i // 4 * 4 + 4]] - 1.0)
        q = 29
        while four.max() * 2.0 ** q > 2.0 ** 31 - 2 or four.sum(1).max() * 2.0 ** q + K > 2.0 ** 33:
            q -= 1
        # words of C (2^-61 S) and of e - 1 (2^-(q + 31), times at most 2 S), dropped products, the sum's unit twice
        words = four[i % 4].sum() * 2.0 ** -61 + 2.0 ** -(q + 30) + K * 2.0 ** -(q + 32) + 2.0 ** -(q + 30)
        bound = words * np.ldexp(1.0, ex) / np.abs(M) + 2.0 ** -52
        err = np.abs((out[r] - M * C[s]) / (M * C[s])).astype(np.float64)
        worst, ratio = max(worst, err.max()), max(ratio, (err / bound).max())
    print(f"{config}, largest efficiency {largest}: max error {worst:.2e}, {ratio:.2f} of the bound")
    assert ratio <= 1.0


@pytest.mark.parametrize("config", ["k10", "k53"])
def test_exact_rate_constants(config):
    """Constants, and constants times a whole power of T in elementary reactions, have the bits of their FP64 products, in
    calls of every size; a Troe reaction of such coefficients is as close to long double as its dozen FP64 roundings."""
    import torch
    import combustion_gb300 as cb
    LD = np.longdouble
    m = copy.deepcopy(util.mechanism(config))
    rows = np.flatnonzero(m.model == synthetic.ELEMENTARY)[:8]
    powers = [0.0, -2.0, -1.0, 1.0, 2.0, 3.0, 4.0, 0.0]
    for r, b in zip(rows, powers):
        m.model[r] = synthetic.IRREVERSIBLE
        m.rate[r] = (m.rate[r, 0], b, 0.0)
        s = int(np.flatnonzero(m.reactants[r])[0])
        m.reactants[r] = 0
        m.reactants[r, s] = 1
    m.rate[rows[-1], 0] = 1e60  # capped at the largest 32-bit number
    troe = np.flatnonzero(m.model == synthetic.TROE)[:2]
    for r, b in zip(troe, (0.0, 2.0)):
        m.rate[r], m.k0[r] = (1e3, b, 0.0), (1e4, 1.0, 0.0)
        m.reactants[r], m.products[r] = 0, 0  # one reactant, and a product that is absent
        m.reactants[r, 2] = m.products[r, 3] = 1
    assert m.active() == m.K - 1
    mech = cb.Mechanism(m)
    cells = synthetic.generate_cells(m.K, 64, config, seed=47)
    cells.amounts[3] = 0.0
    Ctot, _, C = concentrations(m, cells)
    T = cells.temperature
    x = np.vstack([cells.pressure_R, T, cells.volume, cells.amounts])
    factor = {0.0: 1.0, -2.0: (1 / T) * (1 / T), -1.0: 1 / T, 1.0: T, 2.0: T * T, 3.0: T * (T * T), 4.0: (T * T) * (T * T)}
    for reps in (1, 20, 152 * 400 // 64 + 1):
        out = torch.empty((m.R, 64 * reps), dtype=torch.float64, device="cuda")
        mech.reaction_rates(dev(np.tile(x, (1, reps))), out)
        mech.synchronize()
        out = out[:, -64:].cpu().numpy()
        for r, b in zip(rows, powers):
            k = np.minimum(factor[b] * m.rate[r, 0], float(np.finfo(np.float32).max))
            assert np.array_equal(out[r], k * C[int(np.flatnonzero(m.reactants[r])[0])]), (b, reps)
        for r, b in zip(troe, (0, 2)):
            M = Ctot + ((m.efficiencies[r].astype(LD) - 1)[:, None] * C).sum(0)
            ki = LD(1) if b == 0 else T.astype(LD) ** 2
            Pr = M * LD(m.k0[r, 0] / m.rate[r, 0]) * T / ki
            a, T3, T1 = (LD(v) for v in m.troe[r, :3])
            lF = np.log((1 - a) * np.exp(-T / T3) + a * np.exp(-T / T1))
            y = np.log(Pr) - LD(67) / 100 * lF - LD(4) / 10 * np.log(LD(10))
            f1 = y / (-LD(14) / 100 * y - LD(127) / 100 * lF + LD(75) / 100 * np.log(LD(10)))
            ref = np.exp(lF / (f1 * f1 + 1)) * m.rate[r, 0] * ki * Pr / (Pr + 1) * C[2]
            err = np.abs((out[r] - ref) / ref).astype(np.float64).max()
            print(f"{config} Troe, T^{b}: max error {err:.2e}")
            assert err <= 4e-15


def test_coherent_traces():
    """Viscosity at 250 species of a main species and traces whose words' low halves all have the sign of their matrix
    words' (in words of 29 low bits, the worst case of what the integer sums drop): as close to long double as FP64 sums,
    6e-16 and the roundings of a dozen operations beside them."""
    import torch
    import combustion_gb300 as cb
    LD = np.longdouble
    m = util.mechanism("k250")
    K, W = m.K, m.molar_mass.astype(LD)
    mech = cb.Mechanism(m)
    T0, mu0, l0 = synthetic.transport_scales(m)
    mech.transport_setup(T0, mu0, l0)
    visc = mech.transport_coefficients()[1].astype(LD) * (np.sqrt(np.sqrt(LD(T0))) / np.sqrt(LD(mu0)))
    va = np.sqrt(1 / np.sqrt(LD(8)) / np.sqrt(1 + W[:, None] / W))
    b = va * (W / W[:, None]) ** LD(0.25)
    word = np.rint(np.ldexp(va * va, 55)).astype(np.int64)  # the largest below 2^54
    assert 2 ** 53 <= word.max() < 2 ** 54
    low = word - ((word + (1 << 28) >> 29) << 29)
    mains = [K - 1, 0, 100, 17]
    x = np.zeros((K + 1, len(mains) * 3))  # sum n, T/T0, n_0 ..
    for i, k in enumerate(mains):
        for j, trace in enumerate((2.0 ** -27, 2.0 ** -28, 2.0 ** -26 * 0.999)):
            X = np.where(low[k] > 0, trace, 0.0)
            X[k] = 1.0
            x[2:, 3 * i + j] = X[:-1]
            s = 0.0
            for v in X[:-1]:
                s = s + v
            x[0, 3 * i + j] = s + X[-1]
    x[1] = 1500.0 / T0
    for reps in (1, 40, 152 * 260 // x.shape[1] + 1):
        large = torch.empty((K + 2, x.shape[1] * reps), dtype=torch.float64, device="cuda")
        mech.transport(dev(np.tile(x, (1, reps))), large)
        mech.synchronize()
        out = large[1, -x.shape[1]:].cpu().numpy()
        for c in range(x.shape[1]):
            n = x[2:, c]
            s = 0.0
            for v in n:
                s = s + v
            X = np.append(n, x[0, c] - s).astype(LD)
            L = np.log(LD(x[1, c]))
            v = (visc * np.array([L ** i for i in range(5)])).sum(1)
            mu = sum(X[k] * v[k] ** 2 / (X * (va[k] + b[k] * v[k] / v) ** 2).sum() for k in range(K) if X[k] > 0)
            err = float(abs((out[c] - np.sqrt(LD(x[1, c])) * mu) / (np.sqrt(LD(x[1, c])) * mu)))
            print(f"main species {mains[c // 3]}, {x.shape[1] * reps} cells: {err:.2e}")
            assert err <= 2e-15


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
def test_ends_of_the_temperatures(config):
    """Rates from 60 to 9,000 K and transport from 100 to 9,000 K, across the ends of the fixed-point form's
    temperatures, in calls of one cell per block, per warp and per thread: against the oracle, one cell having the same
    bits in each."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    scales = synthetic.transport_scales(m)
    mech.transport_setup(*scales)
    o.set_transport(*scales, *mech.transport_coefficients())
    up, T0 = np.nextafter, scales[0]
    ends = [60.0, up(65.0, 0), 65.0, 80.0, up(100.0, 0), 100.0, 136.0, 150.0, up(200.0, 0), 200.0, 3999.0, 4000.0, 5500.0, 7379.0,
            7381.0, up(8192.0, 0), 8192.0, 9000.0]
    ends += [136.0 * (1 - 1e-12), 136.0 * (1 + 1e-12), 7380.0 * (1 - 1e-12), 7380.0 * (1 + 1e-12)]
    n = 48
    cells = synthetic.generate_cells(m.K, n, config, seed=53)
    scale = cells.temperature.copy()
    cells.temperature[:len(ends)] = ends
    cells.temperature[len(ends):] = np.geomspace(61.0, 8900.0, n - len(ends))
    scale /= cells.temperature
    cells.total_amount *= scale
    cells.amounts *= scale
    rin, pin, tin = o.rates_inputs(cells), o.reaction_rates_inputs(cells), o.transport_inputs(cells)
    hot = np.asarray(cells.temperature) >= 100.0  # (the conductivity polynomials have zeros below)
    calls = (("rates", rin, m.active() + 2, o.rates(rin, scale=True), hot | True),
             ("reaction_rates", pin, m.R, o.reaction_rates(pin, scale=True), hot | True),
             ("transport", tin, m.K + 2, o.transport(tin, scale=True), hot))
    reps = {"k10": 64, "k53": 400, "k250": 400}[config] * 152 // n + 1
    for name, x, rows, (ref, sc), cols in calls:
        first = None
        for r in (1, 40, reps):
            t = torch.full((rows, n * r), float("nan"), dtype=torch.float64, device="cuda")
            getattr(mech, name)(dev(np.tile(np.array(x), (1, r))), t)
            mech.synchronize()
            t = t[:, -n:].cpu().numpy()
            first = t if first is None else first
            assert np.array_equal(t, first, equal_nan=True), (name, r)
        e = util.cond_err(first, ref, sc)[:, cols]
        print(f"{config} {name}: max cond err {np.nanmax(e):.2e} (T = {cells.temperature[cols][np.nanargmax(np.nanmax(e, 0))]:g})")
        assert np.array_equal(np.isfinite(first[:, cols]), np.isfinite(ref[:, cols]))
        assert np.nanmax(e) <= util.PLAIN_TOL


def test_hot_and_cold_cells_take_no_longer():
    """Transport of cells at 3,500 to 7,300 K and rates at 105 to 250 K take as long as at ordinary temperatures."""
    import torch
    import combustion_gb300 as cb
    from combustion_gb300 import surrogate as S
    m = util.mechanism("k53")
    mech = cb.Mechanism(m)
    mech.transport_setup(*synthetic.transport_scales(m))
    n = 1 << 18
    x = S.generate_cells(mech, n, S.distribution("k53", seed=5))
    rates = torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda")
    transport = torch.empty((mech.K + 2, n), dtype=torch.float64, device="cuda")

    def at(lo, hi):
        y = x.clone()
        y[2] = torch.linspace(lo, hi, n, dtype=torch.float64, device="cuda")[torch.randperm(n, device="cuda")]
        y[4:] *= x[2] / y[2]
        return y

    def timed(call):
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times))

    inputs = {name: at(*T) for name, T in (("ordinary", (800, 2800)), ("hot", (3500, 7300)), ("cold", (105, 250)))}
    for call, other in (("transport", "hot"), ("rates", "cold")):
        t = {}
        for name in ("ordinary", other):
            c = inputs[name]
            given = torch.cat([(c[0] * c[3] / c[2])[None], (c[2] / 1000.0)[None], c[4:]])
            t[name] = timed((lambda: mech.rates(c, rates)) if call == "rates" else (lambda: mech.transport(given, transport)))
        print(call, {k: round(v, 2) for k, v in t.items()})
        assert t[other] < 1.25 * t["ordinary"]


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
def test_transport_states(config):
    """Transport of non-finite, zero and negative states: NaN where the oracle has NaN, infinity where it has infinity, the
    rest at the plain bar, in calls of every form."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    scales = synthetic.transport_scales(m)
    mech.transport_setup(*scales)
    o.set_transport(*scales, *mech.transport_coefficients())
    n, K = 48, m.K
    x = np.array(o.transport_inputs(synthetic.generate_cells(K, n, config, seed=59)))  # sum n, T/T0, n_0 ..
    states = [(row, v) for row in (0, 1, 2, 2 + K // 2, K) for v in (np.nan, np.inf, -np.inf)]
    states += [(1, -1.0), (1, 0.0), (0, 0.0), (2, -1e-3 * x[0, 0]), (2 + K // 2, 1e200), (0, 1e200)]
    for c, (row, v) in enumerate(states):
        x[row, c] = v
    with np.errstate(all="ignore"):
        ref, sc = o.transport(list(x), scale=True)
    for r in (1, 40, {"k10": 64, "k53": 192, "k250": 520}[config] * 152 // n + 1):
        t = torch.full((K + 2, n * r), 7.0, dtype=torch.float64, device="cuda")
        mech.transport(dev(np.tile(x, (1, r))), t)
        mech.synchronize()
        t = t[:, -n:].cpu().numpy()
        for c in range(n):
            what = f"{n * r} cells, state {states[c] if c < len(states) else 'ordinary'}"
            assert np.array_equal(np.isnan(t[:, c]), np.isnan(ref[:, c])), what
            assert np.array_equal(np.isinf(t[:, c]), np.isinf(ref[:, c])), what
        both = np.isfinite(ref) & np.isfinite(sc)
        assert (util.cond_err(t, ref, sc)[both] <= util.PLAIN_TOL).all()


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("T0", [250.0, 298.15, 3000.0])
def test_other_reference_temperatures(config, T0):
    """Transport with polynomials in ln(T / T0) of other reference temperatures, whose fixed-point range and words differ:
    from 140 to 7,300 K at the plain bar, one cell having the same bits in calls of every form."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    scales = synthetic.transport_scales(m, T0=T0)
    mech.transport_setup(*scales)
    o.set_transport(*scales, *mech.transport_coefficients())
    n = 48
    cells = synthetic.generate_cells(m.K, n, config, seed=61)
    scale = cells.temperature.copy()
    cells.temperature[:] = np.geomspace(140.0, 7300.0, n)
    scale /= cells.temperature
    cells.total_amount *= scale
    cells.amounts *= scale
    x = np.array(o.transport_inputs(cells))
    ref, sc = o.transport(list(x), scale=True)
    first = None
    for r in (1, 40, {"k10": 64, "k53": 192, "k250": 520}[config] * 152 // n + 1):
        t = torch.full((m.K + 2, n * r), float("nan"), dtype=torch.float64, device="cuda")
        mech.transport(dev(np.tile(x, (1, r))), t)
        mech.synchronize()
        t = t[:, -n:].cpu().numpy()
        first = t if first is None else first
        assert np.array_equal(t, first)
    e = util.cond_err(first, ref, sc)
    print(f"{config}, T0 = {T0}: max cond err {e.max():.2e} (T = {cells.temperature[e.max(0).argmax()]:.0f})")
    assert e.max() <= util.PLAIN_TOL
