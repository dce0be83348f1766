"""Double-float mode: rows in pairs of floats, everything else (the nodes' weights, the two
sums, the scales, the payoff and the discount) in double, on the polynomial path as in
the stepped sweeps.  So the path's errors against double sweeps are no larger than the
stepped double-float sweeps' own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", ["uneven", "random"])
def test_errors_are_the_stepped_sweeps(pkg, pricer, batch):
    wl = pkg.workloads
    opts = pkg.Options.from_batch(wl.uneven_batch(30000, 1) if batch == "uneven" else wl.thesis_dataset("1_RAND", 4000, seed=3))
    rates, days = wl.yield_curve()
    y = pkg.Yield(rates, days)
    exact = pricer.price(opts, y, pkg.BATCHED_FP64, big_threshold=1)
    some = exact > 1e-3

    def error(prices):
        return np.sqrt(np.mean(((prices - exact)[some] / exact[some]) ** 2))

    stepped = error(pricer.price(opts, y, pkg.BATCHED_DF64, big_threshold=1))
    # (a tenth for the accident of two samples of rounding errors)
    assert error(pricer.price(opts, y, pkg.BATCHED_DF64)) <= 1.1 * stepped
