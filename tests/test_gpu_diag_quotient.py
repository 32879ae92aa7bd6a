"""Division by U's diagonal in the FP64 engine's solves, seen alone through one
scatterer: its amplitude at the origin is 1 / M, to one rounding a component; and
dlogf, (dM/dk) / M, where the reciprocal of the pivot would overflow although the
quotient is an ordinary number."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _error(x, a, b):
    """|x - a / b| / |a / b|"""
    ar, ai, br, bi = (Fraction(float(x)) for x in (a.real, a.imag, b.real, b.imag))
    d = br * br + bi * bi
    qr, qi = (ar * br + ai * bi) / d, (ai * br - ar * bi) / d
    er, ei = Fraction(float(x.real)) - qr, Fraction(float(x.imag)) - qi
    return float((er * er + ei * ei) / (qr * qr + qi * qi)) ** 0.5


def test_reciprocal_to_one_rounding(ms):
    # (the "maximum" model's element is a chain of single products and functions, the same
    # bits wherever it is evaluated)
    med = ms.Medium(3, 1, pos=np.zeros(3))
    rng = np.random.default_rng(11)
    ks = rng.uniform(0.3, 6.0, 1500) - 1j * rng.uniform(-3.0, 3.0, 1500)
    _, amps, st = ms.amplitude_batch([med], ks)
    assert np.all(st == 0)
    err = [_error(a[0], np.complex128(1), ms.build_ms_matrix(med, k)[0, 0]) for a, k in zip(amps, ks)]
    # one rounding a component, the rest of order 2^-106
    assert max(err) <= 2.0 ** -53 * (1 + 1e-6)


def test_reciprocal_beyond_the_range(ms):
    # F^-1 of a hard sphere falls as e^{-2 Im k a}: here 1e-310, its derivative 2 a times that
    med = ms.Medium(3, 1, seed=1, model="hardsphere", params=(1000.0,))
    k = 0.5 + 0.35665j
    m, dm = ms.build_ms_matrix(med, k)[0, 0], ms.build_ms_matrix(med, k, deriv=True)[0, 0]
    assert 0 < max(abs(m.real), abs(m.imag)) < 5e-309
    got, st = ms.dk_log_det_batch([med], [k])
    assert st[0] == 0
    # a pivot of 46 bits or fewer: one spacing, 2^-1074, where another kernel rounds its
    # element, one or two in the division
    tol = 8 * 2.0 ** -1074 / abs(m) + 4 * 2.0 ** -53
    assert _error(got[0], dm, m) <= tol
