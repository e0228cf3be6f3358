"""Accuracy of the plain kernels' fixed-point functions on the GPU, one by one, against long double (64-bit mantissa on
x86-64, 113-bit on aarch64).

The bars follow from the functions' words. Relative to the result's last place (ulp, 2^-52 of its power of two):
  2^x    relative 2^-51, a step of its argument, and half an ulp as a double
  log2   a multiple of 2^-51, terms below 2^-59: 2^-52 (1 + 1/64), and half an ulp as a double
  1 / d  a word of 2^-56 or more, truncated: up to 2^-55 of the result below it, and half an ulp
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def run(which, x):
    import torch
    import combustion_gb300 as cb
    return cb.debug_fixed_math(which, torch.from_numpy(np.ascontiguousarray(x)).cuda()).cpu().numpy()


def ulp(v):
    return np.ldexp(LD(1), np.frexp(np.abs(v))[1] - 53)


def test_exp2():
    rng = np.random.default_rng(0)
    q = 2.0 ** -51
    x = np.concatenate([rng.uniform(-1, 1, 1 << 19), np.arange(-1021, 1021) + 0.0, rng.uniform(-1e-6, 1e-6, 1 << 16),
                        (np.arange(-4096, 4096) / 1024.0)[:, None].repeat(3, 1).ravel() + np.tile([-q, 0.0, q], 8192)])
    x = np.rint(x / q) * q  # multiples of 2^-51
    wide = rng.uniform(-1021, 1023, 1 << 18)
    wide = np.rint(wide * 2.0 ** 42) * 2.0 ** -42
    x = np.concatenate([x, wide])
    ref = np.exp2(x.astype(LD))
    err = np.abs(run("exp2", x) - ref)
    ulps = (err / ulp(ref)).astype(float)
    print(f"2^x: {ulps.max():.4f} ulp, rms {np.sqrt((ulps ** 2).mean()):.4f}")
    assert (err <= ref * LD(2) ** -51 + ulp(ref) / 2).all()
    special = np.array([np.inf, -np.inf, np.nan, 1024.0, -1100.0, -1040.0, 0.0, -0.0])
    np.testing.assert_array_equal(run("exp2", special), np.exp2(special))


def test_log2():
    rng = np.random.default_rng(1)
    x = np.concatenate([2.0 ** rng.uniform(-1021, 1023, 1 << 18), rng.uniform(0.5, 2.0, 1 << 19), rng.uniform(65.0, 8192.0, 1 << 18),
                        1.0 + rng.uniform(-1e-3, 1e-3, 1 << 16), 2.0 ** np.arange(-1021, 1023),
                        (1.0 + np.arange(512) / 512.0)[:, None].repeat(3, 1).ravel() * np.tile([1 - 2.0 ** -52, 1.0, 1 + 2.0 ** -52], 512)])
    ref = np.log2(x.astype(LD))
    err = np.abs(run("log2", x) - ref)
    bar = LD(2) ** -52 * (1 + LD(2) ** -6) + ulp(np.maximum(np.abs(ref), 2.0 ** -60)) / 2
    print(f"log2: {float((err / bar).max()):.4f} of the bar")
    assert (err <= bar).all()
    special = np.array([0.0, -0.0, -1.0, np.inf, np.nan, 5e-324, 1.0])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(run("log2", special), np.log2(special))


def test_reciprocal():
    rng = np.random.default_rng(2)
    x = np.concatenate([2.0 ** rng.uniform(-5, 0, 1 << 20), np.nextafter(2.0 ** -np.arange(0, 5.0), 0), 2.0 ** -np.arange(1, 6.0)])
    x = np.rint(x * 2.0 ** 57) * 2.0 ** -57
    ref = 1 / x.astype(LD)
    err = (np.abs(run("rcp", x) - ref) / ulp(ref)).astype(float)
    print(f"1 / d: {err.max():.4f} ulp")
    assert err.max() <= 0.5 + 2.0 ** -55 / 2.0 ** -53 + 0.02


def test_conversions():
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(-512, 512, 1 << 18), rng.uniform(-1, 1, 1 << 18) * 2.0 ** rng.uniform(-60, 0, 1 << 18),
                        [0.0, -0.0, 2.0 ** -51, -(2.0 ** -51), 2.0 ** -52, 2.0 ** -53, 511.999, 1e-300, -1e-300]])
    y = run("fix", x)
    err = np.abs(y - x.astype(LD))
    assert (err <= LD(2) ** -52).all()  # (a value of 2 or more has no bits below, and is itself)
    assert (y.astype(LD) * LD(2) ** 51 == np.rint(y.astype(LD) * LD(2) ** 51)).all()
    assert np.array_equal(y[np.abs(x) >= 2], x[np.abs(x) >= 2])


@pytest.mark.parametrize("config, n", [("k10", 2048), ("k53", 1024), ("k250", 128)])
def test_errors_against_long_double(config, n):
    """Rates and transport of seeded cells against long double: the condition-scaled rms error of every output group is
    below that of the same program in FP64 (the oracle)."""
    import torch
    import combustion_gb300 as cb
    import numpy_restatement
    import oracle
    import util
    from combustion_gb300 import synthetic
    m = util.mechanism(config)
    mech, o = cb.Mechanism(m), oracle.Oracle(m)
    scales = synthetic.transport_scales(m)
    mech.transport_setup(*scales)
    coefs = mech.transport_coefficients()
    o.set_transport(*scales, *coefs)
    cells = synthetic.generate_cells(m.K, n, config, seed=77)
    rin, tin = o.rates_inputs(cells), o.transport_inputs(cells)
    wide = [x.astype(LD) for x in rin]
    wide[1] = 1 / wide[0]
    dev = lambda x: torch.tensor(np.array(x), dtype=torch.float64, device="cuda")  # noqa: E731
    rates = torch.empty((mech.A + 2, n), dtype=torch.float64, device="cuda")
    transport = torch.empty((mech.K + 2, n), dtype=torch.float64, device="cuda")
    mech.rates(dev(rin), rates)
    mech.transport(dev(tin), transport)
    mech.synchronize()
    cases = (("rates", rates, o.rates(rin, scale=True), util.RATES_GROUPS,
              numpy_restatement.rates(m, wide[0], wide[1], wide[2], wide[3], wide[4:])),
             ("transport", transport, o.transport(tin, scale=True), util.TRANSPORT_GROUPS,
              numpy_restatement.transport(m, scales, coefs, tin[0].astype(LD), tin[1].astype(LD), [x.astype(LD) for x in tin[2:]])))
    for name, out, (fp64, scale), groups, ref in cases:
        ours, theirs = (np.abs((x.astype(LD) - ref) / scale).astype(float) for x in (out.cpu().numpy(), fp64))
        for group, rows in groups:
            a, b = (np.sqrt((e[rows] ** 2).mean()) for e in (ours, theirs))
            print(f"{config} {name} {group}: rms {a:.2e} (FP64 {b:.2e}), max {ours[rows].max():.2e} ({theirs[rows].max():.2e})")
            assert a <= b
