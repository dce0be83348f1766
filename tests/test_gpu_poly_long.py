"""Double modes on long bonds with weak mean reversion, whose discounting leans over the
whole tree: the state prices' series has to carry the lean of the steps after the payoff
too.  Also trees at the coefficient table's last rows (4,096 steps) and on both sides of
the switch from fixed-point to double rows."""
import numpy as np
import pytest

from conftest import assert_fp64

pytestmark = pytest.mark.gpu


def _options(pkg, T, t, steps, a, sigma, rng, spread=0.1):
    wl = pkg.workloads
    n = len(T)
    strike = wl.forward_bond_price(t, T) * (1.0 + spread * rng.uniform(-1.0, 1.0, n))
    rates, days = wl.yield_curve()
    opts = pkg.Options(strike, T, t, np.full(n, 365), steps, a, sigma, np.arange(n) % 2)
    return opts, pkg.Yield(rates, days)


def _long_bonds(pkg):
    rng = np.random.default_rng(21)
    n = 1000
    T = rng.uniform(5.0, 50.0, n)
    t = T * rng.uniform(0.05, 0.95, n)
    a = np.exp(rng.uniform(np.log(0.001), np.log(0.05), n))
    sigma = rng.uniform(0.005, 0.03, n)
    # calls and puts at the money that missed the bound by factors of 3 to 11
    T[:6], t[:6] = [48, 48, 45, 45, 50, 50], [24, 24, 20, 20, 25, 25]
    a[:6], sigma[:6] = [0.002, 0.002, 0.002, 0.002, 0.005, 0.005], [0.02, 0.02, 0.025, 0.025, 0.025, 0.025]
    return _options(pkg, T, t, np.full(n, 12), a, sigma, rng)


def _tall_trees(pkg):
    rng = np.random.default_rng(22)
    steps = np.array([60, 60, 60, 60, 96, 96, 24, 24])
    n = np.array([4094, 4095, 4096, 4097, 4096, 4000, 1024, 1025])
    T = (n + 0.5) / steps
    a = np.array([0.05, 0.05, 0.05, 0.05, 0.08, 0.03, 0.03, 0.03])
    return _options(pkg, T, T * 0.4, steps, a, np.full(len(n), 0.01), rng)


def _switch(pkg):
    """n log_top around 5: log_top = (dr dt / M)^2 / 6 is proportional to sigma^2."""
    rng = np.random.default_rng(23)
    n = 120
    T = rng.uniform(10.0, 30.0, n)
    a = rng.uniform(0.01, 0.04, n)
    steps, dt = 12, 1.0 / 12
    dr = np.sqrt(3.0 * (1.0 - np.exp(-2.0 * a * dt)) / (2.0 * a))
    unit = np.floor(T * steps) * (dr * dt / (np.exp(-a * dt) - 1.0)) ** 2 / 6.0
    sigma = np.sqrt(5.0 * np.tile([0.3, 0.97, 1.03, 2.0], n // 4) / unit)
    keep = sigma < 0.03
    return _options(pkg, T[keep], T[keep] * rng.uniform(0.2, 0.8, keep.sum()), np.full(keep.sum(), steps), a[keep],
                    sigma[keep], rng)


def _within_floats(pkg, opts):
    """Trees whose bond values stay within float's exponents at the outermost node, where
    they lean to exp(J dr dt (1 - exp(-a dt n)) / (a dt)): double-float rows hold no others
    (stepped through, they overflow to NaN)."""
    s = pkg.shape(opts)
    dt, a = 1.0 / opts.TermStepCounts, opts.ReversionRates
    dr = opts.Volatilities * np.sqrt(3.0 * (1.0 - np.exp(-2.0 * a * dt)) / (2.0 * a))
    return np.minimum(s["jmax"], s["height"]) * dr * (1.0 - np.exp(-a * dt * s["height"])) / a < 75.0


@pytest.mark.parametrize("batch", [_long_bonds, _tall_trees, _switch])
def test_double_modes_match_oracle(pkg, orc, pricer, batch):
    opts, y = batch(pkg)
    ref = orc.price(opts, y, "f64")
    assert_fp64(pricer.price(opts, y, pkg.BATCHED_FP64), ref, "BATCHED_FP64")
    held = _within_floats(pkg, opts)
    assert held.sum() > 0.6 * opts.N
    assert_fp64(pricer.price(opts, y, pkg.BATCHED_DF64)[held], ref[held], "BATCHED_DF64")
