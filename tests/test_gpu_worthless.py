"""Options that pay at no node of the tree are worth exactly nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64"])
def test_worthless_options_are_zero(pkg, orc, pricer, mode_name):
    """Strikes past the tree's last node: no value anywhere, as the oracle has it."""
    wl = pkg.workloads
    rng = np.random.default_rng(42)
    n = 400
    steps = np.full(n, 12)
    t = rng.uniform(1.0, 6.0, n)
    T = t + rng.uniform(1.0, 4.0, n)
    a = np.asarray(wl.reversion_rate_for_width(rng.integers(3, 24, n) * 2 + 1, 12), dtype=np.float64)
    put = np.arange(n) % 2
    strike = wl.forward_bond_price(t, T) * np.exp(np.where(put == 1, -1.0, 1.0) * rng.uniform(0.05, 0.8, n))
    rates, days = wl.yield_curve()
    opts = pkg.Options(strike, T, t, np.full(n, 365), steps, a, np.full(n, 0.01), put)
    y = pkg.Yield(rates, days)
    ref = orc.price(opts, y, "f64")
    got = pricer.price(opts, y, getattr(pkg, mode_name))
    assert (ref == 0.0).sum() > 100
    assert np.all(got[ref == 0.0] == 0.0)
    assert np.all(got >= 0.0)
