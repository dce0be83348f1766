"""Mean reversion down to the weakest the pricer accepts (a dt = 2e-10): the nodes the
paths visit, the polynomials' degrees and the payoff's place are computed in float, where
1 - exp(-x) of such a rate has no digits left."""
import numpy as np
import pytest

from conftest import assert_fp64, assert_lowp

pytestmark = pytest.mark.gpu


def _tree(X, T, t, steps, a, sigma, put, disc):
    """The tree's price in 64 bits, on the |j| <= n its paths reach (all far inside jmax,
    at whose width the oracle would allocate its rows): state prices at the payoff step
    and bond values there, the drift from the curve's discounts."""
    dt = 1.0 / steps
    n, m = int(T * steps), int(t / dt)
    dr = np.sqrt(3.0 * (sigma * sigma * (1.0 - np.exp(-2.0 * a * dt)) / (2.0 * a)))
    j = np.arange(-n, n + 1)
    x = j * (np.exp(-a * dt) - 1.0)
    up, dn, mid = 1 / 6 + (x * x + x) / 2, 1 / 6 + (x * x - x) / 2, 2 / 3 - x * x
    G = np.exp(-j * dr * dt)
    q, c = (j == 0).astype(float), np.ones(2 * n + 1)
    for _ in range(m):
        g = q * G
        q = mid * g
        q[1:] += (up * g)[:-1]
        q[:-1] += (dn * g)[1:]
    for _ in range(n - m):
        v = mid * c
        v[:-1] += up[:-1] * c[1:]
        v[1:] += dn[1:] * c[:-1]
        c = G * v
    bond = 100.0 * disc(n * dt) / disc(m * dt) * q.sum() / (q @ c) * c
    return disc(m * dt) * (q @ np.maximum(X - bond if put else bond - X, 0.0)) / q.sum()


@pytest.fixture(scope="module")
def batch(pkg):
    wl = pkg.workloads
    rng = np.random.default_rng(31)
    steps = 12
    rows = [(adt, n) for adt in np.geomspace(2e-10, 1e-6, 12) for n in (10, 17, 24, 47, 80)]
    adt, n = (np.array(v) for v in zip(*rows))
    T = (n + 0.5) / steps
    t = T * rng.uniform(0.2, 0.8, len(n))
    rates, days = wl.yield_curve()
    opts = pkg.Options(wl.forward_bond_price(t, T) * rng.uniform(0.99, 1.01, len(n)), T, t, np.full(len(n), 365),
                       np.full(len(n), steps), adt * steps, rng.uniform(0.005, 0.02, len(n)), np.arange(len(n)) % 2)

    def disc(k):
        return np.exp(-wl._curve_rate(k, rates, days) * k)

    ref = [_tree(opts.StrikePrices[i], T[i], t[i], steps, opts.ReversionRates[i], opts.Volatilities[i], opts.Types[i], disc)
           for i in range(len(n))]
    return opts, pkg.Yield(rates, days), np.array(ref)


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64"])
def test_double_modes(pkg, pricer, batch, mode_name):
    """Against the stepped sweeps, and against the tree in 64 bits, where an ulp of exp(-2 a
    dt) moves the rate step, and the price with it, by 2^-53 / (2 a dt) of itself."""
    opts, y, ref = batch
    mode = getattr(pkg, mode_name)
    got = pricer.price(opts, y, mode)
    assert_fp64(got, pricer.price(opts, y, mode, big_threshold=1), mode_name)
    adt = opts.ReversionRates / opts.TermStepCounts
    assert np.all(np.abs(got - ref) <= (1e-10 + 2.0 ** -51 / adt) * ref + 1e-12)


@pytest.mark.parametrize("mode_name", ["BATCHED_FP32", "BATCHED_MIXED"])
def test_float_modes(pkg, pricer, batch, mode_name):
    """Against the tree in 64 bits, and against the uncut trees (sums that are exact to 2^-48)."""
    opts, y, ref = batch
    mode = getattr(pkg, mode_name)
    cut = pricer.price(opts, y, mode)
    assert_lowp(cut, ref, mode_name)
    assert np.max(np.abs(cut - pricer.price(opts, y, mode, big_threshold=1024))) <= 100 * 2.0 ** -46
