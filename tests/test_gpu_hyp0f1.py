"""Rounding of the 0F1 series behind I_d(k, r) for |k| r < 3, as the ratio
I_3(k, r) / I_3(k, 1e-9), from which the prefactor drops out: sin(kr) / (kr), with an
error no larger than the same operations in plain double arithmetic have."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _series(z):
    """regularised 0F1(; 3/2; z), a quotient a term"""
    a, t = 1.5, complex(2.0 / np.sqrt(np.pi))
    s = t
    for i in range(1, 51):
        t = t * z / (i * a)
        s += t
        a += 1.0
        if abs(t) < 1e-16 * abs(s):
            break
    return s


def test_error_of_the_series(ms):
    rng = np.random.default_rng(0)
    ks = rng.uniform(0.1, 2.9, 6000) * np.exp(1j * rng.uniform(-1, 1, 6000))
    near, far = np.full(6000, 1e-9), np.ones(6000)
    got = ms.eval_special(2, 3, ks, far) / ms.eval_special(2, 3, ks, near)
    x = ks.astype(np.clongdouble)
    want = np.sin(x) / x
    c = 0.25 * ks  # a stand-in for the prefactor
    plain = np.array([complex(q) * _series(complex(-(k * k) / 4)) / (complex(q) * _series(complex(-(k * k) * 1e-18 / 4)))
                      for q, k in zip(c, ks)])
    rms = [np.sqrt(np.mean(np.abs((v - want) / want).astype(float) ** 2)) for v in (got, plain)]
    assert rms[0] <= 1.04 * rms[1]
