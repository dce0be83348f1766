"""Busy times of the tail-imbalance statistic: an SM works no longer than the pricing takes,
also where two kernels share the SMs."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64", "BATCHED_MIXED", "BATCHED_FP32"])
def test_busy_times_fit_the_pricing(pkg, pricer, mode_name):
    wl = pkg.workloads
    rates, days = wl.yield_curve()
    y = pkg.Yield(rates, days)
    mode = getattr(pkg, mode_name)
    for batch in (wl.skewed_batch(20000, 2), wl.uneven_batch(5000, 3)):
        opts = pkg.Options.from_batch(batch)
        for _ in range(3):
            pricer.price(opts, y, mode, record_busy=True)
            s = pricer.last_stats
            # (the events bracket the kernels from outside; 20 us for the clocks' steps)
            assert 0.0 < s.busy_mean_ms <= s.busy_max_ms <= s.pricing_ms + 0.02, (s.busy_mean_ms, s.busy_max_ms, s.pricing_ms)
