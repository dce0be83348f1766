"""Host arrays at addresses that are no multiple of their elements' size (fields read out
of a byte buffer): accepted and copied, never loaded in place by a kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = (("strike", "StrikePrices"), ("bond_maturity", "Maturities"), ("option_maturity", "Lengths"),
          ("term_unit", "TermUnits"), ("term_steps", "TermStepCounts"), ("a", "ReversionRates"),
          ("sigma", "Volatilities"), ("type", "Types"))


def _shifted(array, offset):
    """A copy of the array that starts `offset` bytes past an aligned address."""
    raw = np.empty(array.nbytes + 64, dtype=np.uint8)
    start = -raw.ctypes.data % 16 + offset
    view = raw[start:start + array.nbytes].view(array.dtype)
    view[:] = array
    return view


def _case(pkg, n):
    opts = pkg.Options.from_batch(pkg.workloads.uneven_batch(n, 61))
    rates, days = pkg.workloads.yield_curve()
    return opts, pkg.Yield(rates, days)


@pytest.mark.parametrize("n", [1, 37, 5001])
@pytest.mark.parametrize("only", [None, "strike", "term_steps", "sigma"])
def test_pageable_arrays(pkg, pricer, n, only):
    opts, y = _case(pkg, n)
    ref = pricer.price(opts, y, pkg.BATCHED_MIXED)
    odd = pkg.Options(*(_shifted(getattr(opts, f), 1 if only in (None, k) else 0) for k, f in FIELDS))
    assert odd.StrikePrices.ctypes.data % 8 == (1 if only in (None, "strike") else 0)
    out = _shifted(np.zeros(n), 1 if only is None else 0)
    got = pricer.price(odd, y, pkg.BATCHED_MIXED, out=out)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("n", [37, 5001])
def test_pinned_arrays(pkg, pricer, n):
    torch = pytest.importorskip("torch")
    opts, y = _case(pkg, n)
    ref = pricer.price(opts, y, pkg.BATCHED_MIXED)
    keep, ptrs = [], {}
    for k, f in FIELDS:
        a = getattr(opts, f)
        raw = torch.empty(a.nbytes + 64, dtype=torch.uint8).pin_memory()
        raw[1:1 + a.nbytes] = torch.from_numpy(a.view(np.uint8).copy())
        keep.append(raw)
        ptrs[k] = raw.data_ptr() + 1
    out = torch.empty(n, dtype=torch.float64).pin_memory()
    pricer.price_host_ptrs(ptrs, n, y, out.data_ptr(), pkg.BATCHED_MIXED)
    assert np.array_equal(out.numpy(), ref)
