"""Fixed-point rows are taken only where they price as closely as the stepped sweeps: tall
trees with weak reversion, whose uniform error their growth magnifies, are not among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", ["uneven", "tall"])
def test_double_mode_is_as_close_as_the_stepped_sweeps(pkg, pricer, batch):
    wl = pkg.workloads
    if batch == "uneven":
        opts = pkg.Options.from_batch(wl.uneven_batch(5000, 1))
    else:
        b = wl.skewed_batch(100000, 3)
        opts = pkg.Options.from_batch({k: v[b["a"] < 0.05] for k, v in b.items()})
    rates, days = wl.yield_curve()
    y = pkg.Yield(rates, days)
    stepped = pricer.price(opts, y, pkg.BATCHED_FP64, big_threshold=1)
    got = pricer.price(opts, y, pkg.BATCHED_FP64)
    some = stepped > 1e-2
    rel = ((got - stepped)[some] / stepped[some])
    # the stepped sweeps' own error against 80-bit trees is 3.6e-14 (uneven) and 3.5e-14 (tall)
    # of the price; another of that size beside it makes 5e-14
    assert np.sqrt(np.mean(rel * rel)) <= 8e-14
