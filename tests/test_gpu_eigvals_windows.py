"""Eigenvalues of M(k) at sizes around the QR sweep's windows of 30 steps and the
32 rows its searches look at, against numpy's LAPACK on the same matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3])
def test_window_edges(ms, d):
    sizes = [4, 29, 30, 31, 32, 33, 34, 61, 62, 63, 64, 65, 94]
    media = [ms.Medium(d, n, seed=n) for n in sizes]
    for k in (1.3, 2.1 - 0.4j):
        mus, st = ms.eigvals_batch(media, np.full(len(sizes), k + 0j), np.arange(len(sizes), dtype=np.int32))
        assert np.all(st == 0)
        for med, mu in zip(media, mus):
            want = np.linalg.eigvals(ms.build_ms_matrix(med, k))
            # distinct nearest neighbours, within the existing eigenvalue tests' tolerance
            left = list(want)
            for m in mu:
                j = int(np.argmin(np.abs(np.array(left) - m)))
                assert abs(left[j] - m) < 1e-10 * np.abs(want).max()
                left.pop(j)
