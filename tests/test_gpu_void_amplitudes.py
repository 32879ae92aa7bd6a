"""Amplitudes of items that have no result (an entry beyond the mixed engine's
range, a device wait that ran out) read NaN, not what an earlier job left in the
device block the arrays are taken from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

S_RANGE, S_TIMEOUT = 4, 8


def test_range_items(ms):
    n = 70
    med = ms.Medium(3, n, seed=n)
    good = 0.6 + 0.2 * np.arange(6) + 0j
    sig, amps, st = ms.amplitude_batch([med], good, precision="mixed")
    assert np.all(st == 0)
    ks = good.copy()
    ks[1::2] = 0.9 - 40.0j  # e^{|Im k| r} far beyond 1e18
    got, a, st = ms.amplitude_batch([med], ks, precision="mixed")
    assert np.all(st[1::2] & S_RANGE) and np.all(st[0::2] == 0)
    for i in range(6):
        assert np.all(np.isnan(a[i].view(np.float64))) if i % 2 else np.array_equal(a[i], amps[i])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_timed_out_items(ms, precision):
    n = 129
    med = ms.Medium(3, n, seed=n)
    ks = 0.6 + 0.005 * np.arange(400) + 0j  # more items than the device holds at once
    want, amps, st = ms.amplitude_batch([med], ks, precision=precision)
    assert np.all(st == 0)
    ms.debug_first_wait_limit(0)
    try:
        _, a, st = ms.amplitude_batch([med], ks, precision=precision)
    finally:
        ms.debug_first_wait_limit(-1)
    assert np.all(st & S_TIMEOUT)
    assert all(np.all(np.isnan(x.view(np.float64))) for x in a)
    got, a, st = ms.amplitude_batch([med], ks, precision=precision)
    assert np.all(st == 0) and np.array_equal(got, want)
    assert all(np.array_equal(x, y) for x, y in zip(a, amps))
