"""Options far out of the money: the sweeps add non-negative terms, so that a
price keeps its relative accuracy however small it is.  A series or a node cut that is
accurate against the bond's value alone loses these prices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Relative bounds.  The price reacts to an error e of the bond values by about e z / sd, sd
# the log bond price's deviation: below 2,000 e here (z <= 13, sd >= 0.006).  Double rows:
# e about 1e-14 after some hundred steps; double-float rows: 2^-44; oracle in double.
BOUND = {"BATCHED_FP64": 1e-10, "BATCHED_DF64": 1e-9}
SMALLEST = {"BATCHED_FP64": 1e-60, "BATCHED_DF64": 1e-25}  # double-float: float's exponents


@pytest.fixture(scope="module")
def batch(pkg, orc):
    wl = pkg.workloads
    rng = np.random.default_rng(41)
    n = 1500
    steps = rng.integers(6, 25, n)
    t = rng.uniform(1.0, 12.0, n)
    T = t + rng.uniform(1.0, 10.0, n)
    a, sigma = rng.uniform(0.02, 0.15, n), rng.uniform(0.006, 0.02, n)
    put = np.arange(n) % 2
    sd = sigma * (1.0 - np.exp(-a * (T - t))) / a * np.sqrt((1.0 - np.exp(-2.0 * a * t)) / (2.0 * a))
    keep = sd > 0.006
    z = rng.uniform(0.0, 13.0, n) * np.where(put == 1, -1.0, 1.0)
    strike = wl.forward_bond_price(t, T) * np.exp(z * sd)
    rates, days = wl.yield_curve()
    opts = pkg.Options(strike, T, t, np.full(n, 365), steps, a, sigma, put).subset(keep)
    y = pkg.Yield(rates, days)
    return opts, y, orc.price(opts, y, "f64")


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64"])
def test_small_prices_keep_their_digits(pkg, pricer, batch, mode_name):
    opts, y, ref = batch
    got = pricer.price(opts, y, getattr(pkg, mode_name))
    assert np.all(got >= 0.0)
    some = ref > SMALLEST[mode_name]
    assert some.sum() > 800
    rel = np.abs(got - ref)[some] / ref[some]
    assert np.max(rel) <= BOUND[mode_name], (np.max(rel), ref[some][np.argmax(rel)])
    assert np.max(got[~some], initial=0.0) <= 2 * SMALLEST[mode_name]


@pytest.mark.parametrize("mode_name", ["BATCHED_FP32", "BATCHED_MIXED"])
def test_cut_float_trees_keep_small_prices(pkg, pricer, batch, mode_name):
    """The cut leaves out paths of weight exp(-34) of the price, not of the bond: cut and
    uncut prices agree to float rounding at every size that float rows hold."""
    opts, y, ref = batch
    mode = getattr(pkg, mode_name)
    uncut = pricer.price(opts, y, mode, big_threshold=1024)
    cut = pricer.price(opts, y, mode)
    some = uncut > 1e-25
    assert some.sum() > 800
    assert np.max(np.abs(cut - uncut)[some] / uncut[some]) <= 2.0 ** -20
