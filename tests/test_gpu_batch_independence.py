"""An option's price is the same bits whatever batch it is priced in: alone, with a few
others, in a batch that fills the GPU, at any place in it, on one shard or another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("StrikePrices", "Maturities", "Lengths", "TermUnits", "TermStepCounts", "ReversionRates", "Volatilities",
          "Types")


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64", "BATCHED_MIXED", "BATCHED_FP32"])
def test_prices_do_not_depend_on_the_batch(pkg, pricer, mode_name):
    wl = pkg.workloads
    mode = getattr(pkg, mode_name)
    rates, days = wl.yield_curve()
    y = pkg.Yield(rates, days)
    parts = [pkg.Options.from_batch(b) for b in (wl.uneven_batch(900, 5), wl.uniform_book(100, 6),
                                                 wl.skewed_batch(400, 7, heavy_fraction=0.05),
                                                 wl.thesis_dataset("1_RAND", 200, seed=8))]
    base = pkg.Options(*(np.concatenate([getattr(p, f) for p in parts]) for f in FIELDS))
    ref = pricer.price(base, y, mode)
    for idx in (np.arange(base.N)[::-1], np.arange(0, base.N, 43), np.array([0]), np.array([1000, 1200, 1500]),
                np.tile(np.arange(base.N), 12)):
        got = pricer.price(base.subset(idx), y, mode)
        assert np.array_equal(got, ref[idx]), (len(idx), np.max(np.abs(got - ref[idx])))
