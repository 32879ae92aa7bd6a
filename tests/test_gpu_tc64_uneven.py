"""The FP64 engine's tensor-core updates on matrices whose rows of L and columns of
U hold entries of very different size, so that a row maximum times a column maximum
says little about the element they update.  tracelog_lu of such a matrix against a
wider LU, beside the FP64 pipe's own error on the same matrix: a 1 x 1 block of
another size makes the span of the entries too large for the tensor cores and leaves
every operation on the matrix as it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uneven(n, s, seed, p=32):
    """Entries that span just under 2^16 for s = 15.  Identity in the first panel; below it a column of ~1 and a column of zeros, to its
    right a row of zeros and a row of ~1 in the other's place, all else ~2^-s."""
    r = np.random.default_rng(seed)

    def entries(size, *shape):
        return size * (0.75 + 0.25 * r.uniform(size=shape)) * np.exp(2j * np.pi * r.uniform(size=shape))

    m = entries(2.0 ** -s, n, n)
    m[:p, :p] = np.eye(p)
    m[p:, 0], m[p:, 1] = 0.9 * np.exp(2j * np.pi * r.uniform(size=n - p)), 0
    m[0, p:], m[1, p:] = 0, 0.9 * np.exp(2j * np.pi * r.uniform(size=n - p))
    return m * 2.0 ** round(s * (n - p) / n)


def _logdet(m):
    """ln |det| in numpy's widest type, partial pivoting"""
    a = m.astype(np.clongdouble)
    for c in range(len(a)):
        p = c + int(np.argmax(np.abs(a[c:, c])))
        a[[c, p]] = a[[p, c]]
        a[c + 1:, c] /= a[c, c]
        a[c + 1:, c + 1:] -= np.outer(a[c + 1:, c], a[c, c + 1:])
    return np.log(np.abs(np.diag(a))).sum()


@pytest.mark.parametrize("n", [112, 200])
@pytest.mark.parametrize("s", [2, 6, 11, 15])
def test_as_close_as_the_fp64_pipe(ms, n, s):
    tc, pipe = [], []
    for seed in range(8):
        m = _uneven(n, s, seed)
        want = _logdet(m)
        v, info = ms.tracelog_lu(m)
        assert info == 0
        tc.append(float(np.longdouble(v.real) * n - want))
        t = 2.0 ** -30
        big = np.zeros((n + 1, n + 1), dtype=complex)
        big[:n, :n], big[n, n] = m, t
        v, info = ms.tracelog_lu(big)
        assert info == 0
        pipe.append(float(np.longdouble(v.real) * (n + 1) - np.log(np.longdouble(t)) - want))
    # two root mean squares of 8 errors each: a factor 2.5 apart by chance once in a hundred
    # times (F distribution); and the roundings of the result itself, one of them n times 2^-53
    rms = [np.sqrt(np.mean(np.square(x))) for x in (tc, pipe)]
    assert rms[0] <= 2.5 * rms[1] + n * 2.0 ** -53


def test_zero_blocks_and_singular(ms):
    n = 160
    r = np.random.default_rng(5)
    a = r.normal(size=(n, n)) + 1j * r.normal(size=(n, n))
    blocks = np.zeros_like(a)
    for i in range(0, n, 40):
        blocks[i:i + 40, i:i + 40] = a[i:i + 40, i:i + 40]
    got, info = ms.tracelog_lu(blocks)
    want = sum(np.linalg.slogdet(a[i:i + 40, i:i + 40])[1] for i in range(0, n, 40)) / n
    assert info == 0 and abs(got.real - want) < 1e-12
    zero = a.copy()
    zero[:, 100] = 0
    got, info = ms.tracelog_lu(zero)
    assert info == 101 and got.real == -np.inf
    twice = a.copy()
    twice[:, 130] = twice[:, 7]
    got, info = ms.tracelog_lu(twice)
    # a pivot of rounding size, or zero: its logarithm is 30 or more below the others'
    assert got.real < np.linalg.slogdet(a)[1] / n - 30 / n
