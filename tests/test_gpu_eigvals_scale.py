"""Eigenvalues of matrices whose entries' squares leave the exponent range: a
resonant model at its pole (a zero diagonal) and scatterers so far apart that
e^{-Im k r} is of order 1e-170, against numpy's LAPACK on the same matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side", [(2, 390.0), (3, 390.0), (4, 390.0), (4, 350.0), (4, 200.0)])
def test_tiny_entries(ms, n, side):
    tetra = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]]) / np.sqrt(8.0)
    pos = side * tetra[:n] + 0.5 * np.random.default_rng(3).uniform(-1, 1, (n, 3))
    med = ms.Medium(3, n, pos=pos, model="resonant", params=(0.0, 1.0))
    m = ms.build_ms_matrix(med, 1j)
    assert np.all(np.diag(m) == 0) and 0 < np.abs(m).max() < 1e-80
    mus, st = ms.eigvals_batch([med], np.array([1j]))
    assert st[0] == 0
    # numpy's own working on the matrix scaled to 1 by a power of two
    sc = 2.0 ** -np.floor(np.log2(np.abs(m).max()))
    left = list(np.linalg.eigvals(sc * m))
    for mu in sc * mus[0]:
        j = int(np.argmin(np.abs(np.array(left) - mu)))
        assert abs(left[j] - mu) < 1e-10 * np.abs(np.linalg.eigvals(sc * m)).max()
        left.pop(j)
