"""The FP64 engine's trailing updates on the tensor cores (items of n > 96), at
the edges of its panels (32), tiles (128 x 32) and of the dispatch: against the
oracle within the FP64 parity tests' tolerance, and the same whatever the team
and the batch; a matrix whose entries span more than the fixed point serves
(d = 2 far below the axis) takes the FP64 pipe's update."""
import numpy as np
import pytest

from helpers import branch_distance, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(3, 96), (3, 97), (3, 128), (3, 129), (3, 161), (3, 289), (2, 190)])
def test_edges_and_teams(ms, oracle, d, n):
    med = ms.Medium(d, n, seed=n)
    ks = 0.6 + 2.3 * np.arange(200) / 199 - 0.1j
    got, st = ms.tracelog_batch([med], ks)
    assert np.all(st == 0)
    for i in (0, 99):
        one, _ = ms.tracelog_batch([med], ks[i:i + 1])
        few, _ = ms.tracelog_batch([med], ks[i:i + 20])
        assert one[0] == got[i] and np.array_equal(few, got[i:i + 20])
    pick = [0, 99, 199]
    want, _ = oracle.tracelog_batch(d, n, med.pos, ks[pick])
    assert np.max(rel(got[pick].real, want.real)) < 1e-11
    assert np.max(branch_distance(got[pick].imag, want.imag, n)) < 1e-9
    dl, st = ms.dk_log_det_batch([med], ks[:40])
    dl1, _ = ms.dk_log_det_batch([med], ks[7:8])
    assert np.all(st == 0) and dl1[0] == dl[7]
    # the finite difference of the diagonal (step 1e-4) leaves ~1e-12 in both
    assert rel(dl[7], oracle.dk_log_det(d, n, med.pos, ks[7])) < 1e-9
    sig, amps, st = ms.amplitude_batch([med], ks[:3].real)
    m = ms.build_ms_matrix(med, ks[1].real)
    phi = np.exp(1j * ks[1].real * med.pos.reshape(n, d)[:, 0])
    assert np.all(st == 0) and np.max(np.abs(m @ amps[1] - phi)) < 1e-11


def test_wide_span_matches_oracle(ms, oracle):
    med = ms.Medium(2, 300, seed=8)
    ks = np.array([0.7 - 0.8j, 1.4 - 0.9j])  # e^{|Im k| r} over a disk of radius 9.8: entries span > 2^16
    m = np.abs(ms.build_ms_matrix(med, ks[0]))
    assert m.max() / m.min() > 2.0 ** 17
    got, st = ms.tracelog_batch([med], ks)
    want, _ = oracle.tracelog_batch(2, 300, med.pos, ks)
    # cond(M) grows with the span: 1e-9 as the determinant's own sensitivity allows there
    assert np.all(st == 0) and np.max(rel(got.real, want.real)) < 1e-9
