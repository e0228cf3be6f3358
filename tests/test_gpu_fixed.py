"""The plain rates kernels' fixed-point form at the edges of its range, against the FP64 oracle.

Cells at and around the temperatures where a cell changes form (200 K, 8,192 K: the FP64 form outside) or
table piece (2,048 K), in one call with ordinary ones; reactions of every shape (one to four factors on a
side, multiplicities up to three, one to seven net species, every net order, irreversible); a mechanism whose
constants are out of range (the FP64 kernel); calls of 1 cell to more than two waves.
The bar is the plain form's: 1e-12 condition-scaled.
"""
import copy
import os

import numpy as np
import pytest

import util
from combustion_gb300 import synthetic

pytestmark = pytest.mark.gpu
NTHREADS = os.cpu_count() or 4


def shapes_mechanism(config):
    """The generator's mechanism with reactions of the shapes it never draws."""
    m = copy.deepcopy(util.mechanism(config))
    K = m.K
    sides = [  # reactants, products (species index: multiplicity); net order within -1 .. 2
        ({0: 3}, {1: 1, 2: 1, 3: 1}), ({0: 1, 1: 1, 2: 1}, {3: 2, 4: 1}), ({2: 2, 3: 1, 4: 1}, {5: 1, 6: 1, 7: 1}),
        ({5: 1}, {6: 2}), ({6: 1}, {5: 1, 7: 1, 8: 1}), ({7: 2}, {8: 1}), ({1: 1, K - 1: 1}, {2: 1, K - 1: 1}),
        ({0: 1, 1: 1, 2: 1, 3: 1}, {4: 1, 5: 1, 6: 2}), ({8: 1}, {7: 1}), ({4: 2}, {0: 2})]
    kinds = [np.flatnonzero(m.model == k) for k in (synthetic.ELEMENTARY, synthetic.THREE_BODY, synthetic.TROE)]
    rows = list(kinds[0][:len(sides)]) + [kinds[1][0], kinds[2][0]]
    for r, (lhs, rhs) in zip(rows, sides + [sides[1], sides[4]]):
        m.reactants[r] = 0
        m.products[r] = 0
        for k, n in lhs.items():
            m.reactants[r, k] = n
        for k, n in rhs.items():
            m.products[r, k] = n
    m.model[rows[2]] = synthetic.IRREVERSIBLE
    lin = kinds[0][len(sides)]
    m.model[lin] = synthetic.LINDEMANN
    m.k0[lin] = (m.rate[lin, 0] * 1e-3, m.rate[lin, 1] - 0.3, m.rate[lin, 2] * 0.7)
    m.efficiencies[lin] = np.linspace(0.5, 4.0, K)
    m.meta = {"config": config + "-shapes"}
    assert m.active() == K - 1
    return m


def out_of_range_mechanism(config):
    m = copy.deepcopy(util.mechanism(config))
    m.rate[0] = (1e40, 0.0, 2e5)
    return m


def edge_temperatures(config, n):
    cells = synthetic.generate_cells(util.mechanism(config).K, n, config, seed=31)
    up = np.nextafter
    edges = [150.0, up(200.0, 0), 200.0, up(200.0, 1e9), 999.0, 1000.0, up(1000.0, 1e9), up(2048.0, 0), 2048.0,
             up(2048.0, 1e9), 4096.0, up(8192.0, 0), 8192.0, 9000.0]
    scale = cells.temperature.copy()
    cells.temperature[:len(edges)] = edges[:n]
    scale /= cells.temperature  # the ideal-gas total keeps P and V
    cells.total_amount *= scale
    cells.amounts *= scale
    return cells


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("make", [util.mechanism, shapes_mechanism, out_of_range_mechanism],
                         ids=["generator", "shapes", "out-of-range"])
def test_range_and_shapes(config, make):
    import torch
    import combustion_gb300 as cb
    import oracle
    m = make(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    cells = edge_temperatures(config, 96)
    rin = o.rates_inputs(cells)
    dev = lambda x: torch.tensor(np.array(x), dtype=torch.float64, device="cuda")  # noqa: E731
    out = torch.full((mech.A + 2, cells.n), float("nan"), dtype=torch.float64, device="cuda")
    mech.rates(dev(rin), out)
    pin = o.reaction_rates_inputs(cells)
    progress = torch.full((mech.R, cells.n), float("nan"), dtype=torch.float64, device="cuda")
    mech.reaction_rates(dev(pin), progress)
    mech.synchronize()
    for name, x, (ref, sc) in (("rates", out, o.rates(rin, nthreads=NTHREADS, scale=True)),
                               ("progress", progress, o.reaction_rates(pin, nthreads=NTHREADS, scale=True))):
        x = x.cpu().numpy()
        assert np.array_equal(np.isfinite(x), np.isfinite(ref))
        e = util.cond_err(x, ref, sc)
        print(f"{config} {name}: max cond err {np.nanmax(e):.2e} (cell T = {cells.temperature[np.nanargmax(np.nanmax(e, 0))]:g})")
        assert np.nanmax(e) <= util.PLAIN_TOL


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 4865, 155649, 311297])
def test_call_sizes(n):
    """Every launch shape gives each cell the value it has in a call of its own block."""
    import torch
    import combustion_gb300 as cb
    from combustion_gb300 import surrogate as S
    mech = cb.Mechanism(util.mechanism("k10"))
    cells = S.generate_cells(mech, n, S.distribution("k53", seed=9))
    out = torch.full((mech.A + 2, n), float("nan"), dtype=torch.float64, device="cuda")
    mech.rates(cells, out)
    pick = torch.unique(torch.tensor([0, n // 3, n // 2, n - 1], device="cuda"))
    few = torch.empty((mech.A + 2, len(pick)), dtype=torch.float64, device="cuda")
    mech.rates(cells[:, pick].contiguous(), few)
    assert torch.isfinite(out).all()
    scale = out.abs().amax(dim=0)
    assert ((out[:, pick] - few).abs() <= 1e-12 * scale[pick]).all()


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
def test_transport_range_and_forms(config):
    """Transport at the edges of its fixed-point temperatures (200 and 4,000 K), with pure, negative, zero, huge and
    non-finite amounts, against the oracle; and a cell has the same bits in a small call (one cell per warp) as in a
    large one (one per thread)."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    K = m.K
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    scales = synthetic.transport_scales(m)
    mech.transport_setup(*scales)
    o.set_transport(*scales, *mech.transport_coefficients())
    cells = synthetic.generate_cells(K, 64, config, seed=33)
    tin = np.array(o.transport_inputs(cells))  # sum n, T/T0, n_0 ..
    T0 = scales[0]
    edges = [150.0, np.nextafter(200.0, 0), 200.0, 300.0, 1000.0, 3000.0, np.nextafter(4000.0, 0), 4000.0, 5000.0]
    for c, T in enumerate(edges):
        tin[1, c] = T / T0
    c = len(edges)
    tin[2:, c] *= 1e-170            # subnormal products
    tin[0, c] *= 1e-170
    tin[2:, c + 1] *= 1e160
    tin[0, c + 1] *= 1e160
    tin[2, c + 2] = -0.2 * tin[0, c + 2]
    tin[2 + K // 2, c + 3] = 0.0
    tin[2:, c + 4] = 1e-9 * tin[0, c + 4] / K  # the bulk species but for traces
    tin[2:, c + 5] = 1e-9 * tin[0, c + 5] / K  # species 0 but for traces
    tin[2, c + 5] = tin[0, c + 5] * (1.0 - 1e-8)
    dev = lambda x: torch.tensor(x, dtype=torch.float64, device="cuda")  # noqa: E731

    def run(x):
        out = torch.full((K + 2, x.shape[1]), float("nan"), dtype=torch.float64, device="cuda")
        mech.transport(dev(x), out)
        mech.synchronize()
        return out.cpu().numpy()

    small = run(tin)
    ref, sc = o.transport(list(tin), nthreads=NTHREADS, scale=True)
    assert np.array_equal(np.isfinite(small), np.isfinite(ref))
    e = util.cond_err(small, ref, sc)
    print(f"{config} transport: max cond err {np.nanmax(e):.2e} (cell {np.nanargmax(np.nanmax(e, 0))})")
    assert np.nanmax(e) <= util.PLAIN_TOL
    bad = tin.copy()
    bad[2, 0], bad[0, 1], bad[1, 2] = np.nan, np.inf, np.nan
    for x in (tin, bad):  # the same cells in a call of one cell per thread
        reps = {"k10": 64, "k53": 192, "k250": 520}[config] * 152 // 64 + 1
        large = run(np.tile(x, (1, reps)))
        assert np.array_equal(large[:, :64], large[:, -64:], equal_nan=True)
        assert np.array_equal(run(x), large[:, :64], equal_nan=True)


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("make", [util.mechanism, shapes_mechanism], ids=["generator", "shapes"])
def test_rates_small_calls_match_large_ones(config, make):
    """A cell has the same bits in a small call (one cell per warp) as in a large one (one per thread), those that
    take the FP64 form among them (more than a warp's worth)."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = make(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    cells = edge_temperatures(config, 48)
    rin, pin = np.array(o.rates_inputs(cells)), np.array(o.reaction_rates_inputs(cells))
    rin[4, 20] = np.nan
    rin[0, 21] = pin[0, 21] = 0.0
    dev = lambda x: torch.tensor(x, dtype=torch.float64, device="cuda")  # noqa: E731
    reps = {"k10": 64, "k53": 400, "k250": 400}[config] * 152 // 48 + 1
    for call, x, rows in ((mech.rates, rin, mech.A + 2), (mech.reaction_rates, pin, mech.R)):
        out = {}
        for r in (1, 40, reps):
            t = torch.full((rows, 48 * r), float("nan"), dtype=torch.float64, device="cuda")
            call(dev(np.tile(x, (1, r))), t)
            mech.synchronize()
            out[r] = t[:, -48:].cpu().numpy()
        assert np.array_equal(out[1], out[40], equal_nan=True)
        assert np.array_equal(out[1], out[reps], equal_nan=True)


@pytest.mark.parametrize("n", [1, 127, 128, 257, 39000])
def test_surrogate_call_sizes(n):
    """The inference kernel writes the transport properties of every cell of a call and nothing beyond, whatever
    the call's last tile holds; fallback and audited cells (one launch for both lists when few, two otherwise) keep the
    plain kernel's bits."""
    import torch
    import combustion_gb300 as cb
    from combustion_gb300 import surrogate as S
    m = util.mechanism("k10")
    mech = cb.Mechanism(m)
    mech.transport_setup(*synthetic.transport_scales(m))
    s = S.Surrogate(mech, width=256, hidden_layers=2, batch=1024, seed=3)
    s.generate(1 << 13, S.distribution("k10", seed=2))
    cells = S.generate_cells(mech, 39000, S.distribution("k10", seed=7))[:, :n].contiguous()
    cells[2, ::5] = 5000.0  # outside the training range
    full = torch.full((mech.K + 2, n + 130), -1.0, dtype=torch.float64, device="cuda")
    s.transport(cells, full[:, :n], gate=False)
    every = torch.full((mech.K + 2, 39000), -1.0, dtype=torch.float64, device="cuda")
    s.transport(torch.cat([cells, cells.flip(1).repeat(1, 39000 // n + 1)], 1)[:, :39000].contiguous(), every, gate=False)
    assert torch.equal(full[:, :n], every[:, :n])
    assert bool((full[:, n:] == -1.0).all()) and bool((full[:, :n] > 0).all())
    gated = torch.empty((mech.K + 2, n), dtype=torch.float64, device="cuda")
    st = s.transport(cells, gated, audit_stride=3)
    plain = torch.empty_like(gated)
    rates = torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda")
    mech.rates_transport(cells, rates, plain)
    idx = torch.arange(n, device="cuda")
    own = (idx % 5 == 0) | (idx % 3 == 7919 % 3)
    assert st["fallback_cells"] >= int((idx % 5 == 0).sum())
    assert torch.equal(gated[:, own], plain[:, own])


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
def test_mixed_small_calls_match_large_ones(config):
    """The mixed-precision form: a cell has the same bits in calls of 1, 47, 480 and more cells than go one per warp."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = shapes_mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    mech.transport_setup(*synthetic.transport_scales(m))
    cells = edge_temperatures(config, 48)
    x = np.array(o.rates_inputs(cells))
    x[4, 20], x[2, 22], x[3, 23] = np.nan, np.nan, 0.0
    reps = 640 * 152 // 48 + 1
    large = None
    for n in (48 * reps, 480, 47, 1):
        xin = torch.tensor(np.tile(x, (1, n // 48 + 1))[:, :n].copy(), dtype=torch.float64, device="cuda")
        r = torch.full((mech.A + 2, n), float("nan"), dtype=torch.float64, device="cuda")
        t = torch.full((mech.K + 2, n), float("nan"), dtype=torch.float64, device="cuda")
        mech.rates_transport(xin, r, t, mixed=True)
        mech.synchronize()
        both = torch.cat([r, t]).cpu().numpy()
        if large is None:
            large = both[:, -48:]
        assert np.array_equal(both, np.tile(large, (1, n // 48 + 1))[:, :n], equal_nan=True)
    xin = torch.tensor(x, dtype=torch.float64, device="cuda")
    uniform, split = torch.empty_like(r[:, :1]).expand(-1, 48).clone(), torch.empty_like(r[:, :1]).expand(-1, 48).clone()
    mech.rates([xin[0, :1], xin[1, :1]] + list(xin[2:]), uniform, uniform_pressure=True, mixed=True)
    xin[:2] = xin[:2, :1].clone()
    mech.rates(xin, split, mixed=True)
    mech.synchronize()
    assert torch.equal(uniform.nan_to_num(7.0), split.nan_to_num(7.0))


@pytest.mark.parametrize("config", ["k10", "k53", "k250"])
@pytest.mark.parametrize("mixed", [False, True])
def test_fused_call_beside_and_after(config, mixed):
    """Rates and transport of one call, running beside each other or one after the other, give what two calls give;
    where their outputs share memory the transport's are the last written; and the call can be captured."""
    import torch
    import combustion_gb300 as cb
    import oracle
    m = util.mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    mech.transport_setup(*synthetic.transport_scales(m))
    sizes = {"k10": (1, 300, 1000, 5000, 70001), "k53": (1, 300, 10100, 70001), "k250": (1, 456, 1000, 3000, 12001)}[config]
    for n in sizes:
        cells = synthetic.generate_cells(m.K, n, config, seed=7)
        x = torch.tensor(np.array(o.rates_inputs(cells)), dtype=torch.float64, device="cuda")
        new = lambda rows: torch.full((rows, n), float("nan"), dtype=torch.float64, device="cuda")  # noqa: E731
        r, t, alone, shared = new(mech.A + 2), new(mech.K + 2), new(mech.A + 2), new(mech.K + 2)
        mech.rates(x, alone, mixed=mixed)
        mech.rates_transport(x, r, t, mixed=mixed)
        mech.rates_transport(x, shared[:mech.A + 2], shared, mixed=mixed)
        mech.synchronize()
        assert torch.isfinite(r).all() and torch.isfinite(t).all()
        assert torch.equal(r, alone) and torch.equal(shared, t)
        if n == 300:
            r2, t2 = new(mech.A + 2), new(mech.K + 2)
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                mech.rates_transport(x, r2, t2, mixed=mixed)
            for _ in range(3):
                graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(r2, r) and torch.equal(t2, t)
