"""Items beyond the mixed engine's FP32 range (MSGPU_S_RANGE) in a batch whose
matrices are shared by clusters of CTAs: every CTA of a team must see the same
range, also where only one of them holds the large entries, and the batch's other
items must come back as they do without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

S_RANGE = 4


@pytest.mark.parametrize("d,n", [(3, 161), (2, 140)])
def test_out_of_range_items_beside_others(ms, d, n):
    med = ms.Medium(d, n, seed=n)
    x = med.pos.reshape(n, d)
    rmax = np.sqrt(((x[:, None] - x[None, :]) ** 2).sum(-1)).max()
    # e^{|Im k| r} / (4 pi r) passes 1e18 for the farthest pairs only, up to most of them
    far = 0.9 - 1j * np.linspace(44.0, 120.0, 12) / rmax
    good = 0.6 + 0.2 * np.arange(12) - 0.1j
    ks = np.empty(24, dtype=complex)
    ks[0::2], ks[1::2] = far, good
    for batch in (ms.tracelog_batch, ms.dk_log_det_batch, ms.amplitude_batch):
        want, st = batch([med], good, precision="mixed")[::2] if batch is ms.amplitude_batch else batch(
            [med], good, precision="mixed")
        assert np.all(st == 0)
        for _ in range(20):
            got, st = batch([med], ks, precision="mixed")[::2] if batch is ms.amplitude_batch else batch(
                [med], ks, precision="mixed")
            assert np.all(st[1::2] == 0) and np.array_equal(got[1::2], want)
            out = (st[0::2] & S_RANGE) != 0
            assert np.all(out[1:]) and np.all(np.isnan(got[0::2][out].real))
