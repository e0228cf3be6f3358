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
