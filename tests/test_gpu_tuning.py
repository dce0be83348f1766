"""The autotuner times the engine that the configured calls run: a tuned or cached
threshold below the default moves no tree off the paths of an untuned call, and a
whole record handed to a call prices as a context configured with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wide(pkg):
    """Trees 601 to 1,501 nodes wide whose paths stay within some 250."""
    wl = pkg.workloads
    rng = np.random.default_rng(51)
    n = 64
    w = np.tile([601, 801, 1001, 1501], n // 4)
    steps = np.full(n, 96)
    height = rng.integers(500, 900, n)
    T = (height + 0.5) / 96
    t = T * rng.uniform(0.3, 0.7, n)
    rates, days = wl.yield_curve()
    opts = pkg.Options(wl.forward_bond_price(t, T), T, t, np.full(n, 365), steps, wl.reversion_rate_for_width(w, 96),
                       np.full(n, 0.008), np.arange(n) % 2)
    return opts, pkg.Yield(rates, days)


def _layout(p):
    s = p.last_stats
    return s.n_block_trees, s.n_warp_tasks, s.kernel_launches


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64", "BATCHED_MIXED", "BATCHED_FP32"])
@pytest.mark.parametrize("threshold", [256, 512])
def test_cached_threshold_keeps_the_fast_paths(pkg, pricer, tmp_path, mode_name, threshold):
    torch = pytest.importorskip("torch")
    opts, y = _wide(pkg)
    mode = getattr(pkg, mode_name)
    ref = pricer.price(opts, y, mode)
    blocks = pricer.last_stats.n_block_trees
    cache = tmp_path / "tune"
    mask = pricer.get_config(mode).warp_k_mask
    cache.write_text(f"{torch.cuda.get_device_name(0)}|{mode} 128 {threshold} {mask}\n")
    with pkg.Pricer(0, tune_cache=str(cache)) as p:
        assert p.get_config(mode).big_threshold == threshold
        got = p.price(opts, y, mode)
        # no more trees off the warps than the threshold sends there after cutting: the
        # uncut widths would send all of them
        if mode_name in ("BATCHED_FP64", "BATCHED_DF64"):
            assert p.last_stats.n_block_trees == blocks
            assert np.array_equal(got, ref)
        else:
            assert blocks == 0
            assert p.last_stats.n_block_trees < opts.N
            # FP32 sums keep the order of the tuned layout's uncut trees
            uncut = p.price(opts, y, mode, big_threshold=threshold)
            assert p.last_stats.n_block_trees == opts.N
            assert np.max(np.abs(got - uncut)) <= 100 * 2.0 ** -46


@pytest.mark.parametrize("mode_name", ["BATCHED_FP64", "BATCHED_DF64", "BATCHED_MIXED", "BATCHED_FP32"])
def test_whole_record_is_no_limit(pkg, mode_name):
    opts, y = _wide(pkg)
    mode = getattr(pkg, mode_name)
    with pkg.Pricer(0) as p:
        for record in (lambda: p.get_config(mode), lambda: p.autotune(opts, y, mode, repeats=1)):
            best = record()
            plain = p.price(opts, y, mode)
            layout = _layout(p)
            again = p.price(opts, y, mode, block_size=best.block_size, big_threshold=best.big_threshold,
                            warp_k_mask=best.warp_k_mask)
            assert _layout(p) == layout
            assert np.array_equal(plain, again)


def test_noalloc_float_prices_are_the_uncut_trees(pkg, pricer):
    """The allocation-free entry point's threshold (512) leaves K = 32 out of its K set; its
    float trees are cut all the same, with the sums of their uncut layout."""
    import ctypes
    torch = pytest.importorskip("torch")
    opts, y = _wide(pkg)
    arrays = {"strike": opts.StrikePrices, "bond_maturity": opts.Maturities, "option_maturity": opts.Lengths,
              "term_unit": opts.TermUnits.view(np.int16), "term_steps": opts.TermStepCounts.view(np.int16),
              "a": opts.ReversionRates, "sigma": opts.Volatilities, "type": opts.Types}
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in arrays.items()}
    rate, day = torch.from_numpy(y.Prices).cuda(), torch.from_numpy(y.TimeSteps).cuda()
    out = torch.empty(opts.N, dtype=torch.float64, device="cuda")
    c_opts, c_yield = pkg._Options(opts.N, *(t.data_ptr() for t in dev.values())), pkg._Yield(y.N, rate.data_ptr(), day.data_ptr())
    rc = pkg.lib().hwt_price_device_noalloc(ctypes.byref(c_opts), ctypes.byref(c_yield), pkg.BATCHED_FP32, out.data_ptr(), None)
    assert rc == pkg.HWT_OK
    uncut = pricer.price(opts, y, pkg.BATCHED_FP32, block_size=64, big_threshold=512)
    assert np.max(np.abs(out.cpu().numpy() - uncut)) <= 100 * 2.0 ** -46
