"""Matrices shared by a cluster of CTAs: a small batch gives each matrix several
CTAs, a large one gives it one, and an item's result must not depend on it.
Sizes at the edges of panels (32) and update tiles (64), n smaller than the
team; every kind; d = 2 for the grouped assembly."""
import numpy as np
import pytest

from helpers import branch_distance, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(3, 1), (3, 33), (3, 64), (3, 65), (3, 129), (2, 70)])
def test_team_size_does_not_change_results(ms, oracle, d, n):
    med = ms.Medium(d, n, seed=n)
    ks = 0.6 + 2.3 * np.arange(400) / 399 - 0.1j
    pick = [0, 7, 399]
    for batch in (ms.tracelog_batch, ms.dk_log_det_batch):
        many, st = batch([med], ks)
        few, st_few = batch([med], ks[:40])
        assert np.all(st == 0) and np.all(st_few == 0) and np.array_equal(few, many[:40])
        for i in pick:
            one, st1 = batch([med], ks[i:i + 1])
            assert st1[0] == 0 and one[0] == many[i]
    many, amps, _ = ms.amplitude_batch([med], ks.real)
    one, amp1, _ = ms.amplitude_batch([med], ks.real[7:8])
    assert one[0] == many[7] and np.array_equal(amp1[0], amps[7])
    # the FP64 parity tests' tolerance
    got, _ = ms.tracelog_batch([med], ks[pick])
    want, _ = oracle.tracelog_batch(d, n, med.pos, ks[pick])
    assert np.max(rel(got.real, want.real)) < 1e-11
    assert np.max(branch_distance(got.imag, want.imag, n)) < 1e-9


@pytest.mark.parametrize("d,n", [(3, 20), (3, 65), (3, 161), (2, 140)])
def test_mixed_team_size_does_not_change_results(ms, oracle, d, n):
    """The mixed engine's clusters: panels of few rows, columns solved a lane per
    row, tiles and refinement residuals shared; bits equal to one CTA's."""
    med = ms.Medium(d, n, seed=n)
    ks = 0.6 + 2.3 * np.arange(400) / 399 - 0.1j
    for batch in (ms.tracelog_batch, ms.dk_log_det_batch):
        many, st = batch([med], ks, precision="mixed")
        few, st_few = batch([med], ks[:40], precision="mixed")
        one, st1 = batch([med], ks[7:8], precision="mixed")
        assert np.all(st == 0) and np.all(st_few == 0) and st1[0] == 0
        assert np.array_equal(few, many[:40]) and one[0] == many[7]
    many, amps, _ = ms.amplitude_batch([med], ks.real, precision="mixed")
    one, amp1, _ = ms.amplitude_batch([med], ks.real[7:8], precision="mixed")
    assert one[0] == many[7] and np.array_equal(amp1[0], amps[7])
    pick = [0, 7, 399]
    got, _ = ms.tracelog_batch([med], ks[pick], precision="mixed")
    want, _ = oracle.tracelog_batch(d, n, med.pos, ks[pick])
    # the mixed engine's stated bound
    assert np.max(rel(got.real, want.real)) < 1e-8
    assert np.max(branch_distance(got.imag, want.imag, n)) < 1e-6
