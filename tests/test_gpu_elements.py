"""FP64 matrix elements of d = 3 by the tables (sin, cos of j pi/32, 2^(j/32)):
against the oracle over real and complex k of either sign, at the edges of the
reductions and beyond their range (the CUDA functions take over at |k r| = 1e5
and |Im k r| = 690)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0.0, 1.3, -2.7, 3.0 - 0.05j, 0.7 + 0.9j, -1.1 - 3.0j, np.pi / 64, 40.0 - 20.0j,
                               3.0e5, 1.0 + 300.0j])
@pytest.mark.parametrize("deriv", [False, True])
def test_elements_match_oracle(ms, oracle, k, deriv):
    n = 40
    med = ms.Medium(3, n, seed=17)
    got = ms.build_ms_matrix(med, k, deriv=deriv)
    want = oracle.ms_matrix(3, n, med.pos, k, deriv=deriv)
    # the oracle has no value of dG/dk at k = 0, where its formula divides by k
    off = ~np.eye(n, dtype=bool) & np.isfinite(want)
    x = med.pos.reshape(n, 3)
    kr = np.abs(k) * np.sqrt(((x[:, None] - x[None, :]) ** 2).sum(-1))
    # relative, in units of 2^-53: r to 2 on either side (three squares, their sum, a root)
    # and the product k r to 1, times |k r| in the phase and the growth; a few ulp of the rest
    tol = (8.0 * kr + 32.0) * 2.0 ** -53
    err = np.abs(got - want) / np.maximum(np.abs(want), 1e-300)
    assert np.all(err[off] <= tol[off])
