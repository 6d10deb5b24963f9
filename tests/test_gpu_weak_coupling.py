"""Networks whose modes couple weakly: permanents and all-minors in which factors are
far below their largest possible sums (a 50:50 splitter on two modes, coupled by eps to
the rest, both doubly occupied at the output), against Glynn's sum in exact integers.
The sums themselves are rounded once to fixed point (62 bits of the largest possible
sum); the products add nothing but the relative error of 62-bit values."""
import itertools
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BITS = 200  # every entry is a multiple of 2^-200


def _matrix(m, eps, seed):
    rng = np.random.default_rng(seed)
    Q, _ = np.linalg.qr(rng.normal(size=(m - 2, m - 2)) + 1j * rng.normal(size=(m - 2, m - 2)))
    U = np.zeros((m, m), dtype=complex)
    U[:2, :2] = np.array([[1.0, 1.0], [1.0, -1.0]]) * np.sqrt(0.5)
    U[2:, 2:] = Q
    return U + eps * (rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))) / np.sqrt(2.0 * m)


def _exact_matrix(m, eps, seed):
    """The same with entries that fixed point and FP64 sums hold exactly: multiples of 2^-50
    (a row's largest sum is below 8), so that the products' own error is all there is."""
    U = _matrix(m, eps, seed)
    U[:2, :2] *= 0.75 / np.sqrt(0.5)
    return np.round(U * 2.0 ** 50) / 2.0 ** 50


def _int(x):
    v = Fraction(float(x)) * 2 ** BITS
    assert v.denominator == 1
    return v.numerator


def _glynn(U, cols, rows, minors, exact=False):
    """Glynn's sum over the signs of the particles `cols` and the factors `rows`: the
    permanent, or every column's minor; and the bound on its error."""
    n = len(cols)
    E = [[(_int(U[r, c].real), _int(U[r, c].imag)) for c in cols] for r in rows]
    F = U[np.ix_(rows, cols)]
    # the entries' roundings: half a unit each, 2^-61 of the largest possible sum at most
    delta = (0 if exact else n) * np.sqrt(0.5) * 2.0 ** -61 * np.maximum(abs(F.real), abs(F.imag)).sum(axis=1)
    out = [[0, 0] for _ in range(n if minors else 1)]
    tol = 0.0
    for tail in itertools.product((1, -1), repeat=n - 1):
        d = (1,) + tail
        p = (1, 0)
        mag, wide = 1.0, 1.0
        for row, de in zip(E, delta):
            s = (sum(x * k[0] for x, k in zip(d, row)), sum(x * k[1] for x, k in zip(d, row)))
            p = p[0] * s[0] - p[1] * s[1], p[0] * s[1] + p[1] * s[0]
            a = abs(complex(s[0] / 2 ** BITS, s[1] / 2 ** BITS))
            mag *= a
            wide *= a + de
        sg = 1 if d.count(-1) % 2 == 0 else -1
        for i in range(len(out)):
            w = sg * (d[i] if minors else 1)
            out[i][0] += w * p[0]
            out[i][1] += w * p[1]
        # every product 2^-54 of its size per factor, and the FP64 additions (at most 2^6 in a row)
        tol += wide - mag + (len(rows) * 2.0 ** -54 + 2.0 ** -47) * wide
    unit = 2 ** (BITS * len(rows) + n - 1)
    return [complex(Fraction(re, unit), Fraction(im, unit)) for re, im in out], tol / 2.0 ** (n - 1)


@pytest.mark.parametrize("eps", [1.0, 1e-2, 1e-3, 1e-4, 1e-6, 1e-8])
def test_permanents(eps):
    from theboss_gb300 import _native

    m, n = 12, 12
    U = _matrix(m, eps, 12)
    S, T = np.ones(m, dtype=np.int32), np.array([2, 2] + [1] * 8 + [0, 0], dtype=np.int32)
    rows = np.repeat(np.arange(m), T).tolist()
    (ref,), tol = _glynn(U, list(range(n)), rows, False)
    assert tol < 1e-4 * abs(ref)
    got = list(_native.perm_batch(U, S[None, :], T[None, :], _native.CHIN_HUH))
    got += list(_native.perm_batch(U, np.tile(S, (40, 1)), np.tile(T, (40, 1)), _native.CHIN_HUH))  # rows made on the GPU
    for g in got:
        assert abs(g - ref) <= tol, (eps, g, ref, abs(g - ref) / abs(ref), tol / abs(ref))
    # Glynn's form takes the outputs' signs here (fewer codes), whose products do not vanish with eps
    (ref,), tol = _glynn(U.T.copy(), rows, list(range(n)), False)
    got = _native.perm_batch(U, S[None, :], T[None, :], _native.GLYNN)[0]
    assert abs(got - ref) <= tol, (eps, got, ref, abs(got - ref) / abs(ref), tol / abs(ref))


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-5, 1e-7])
def test_minors(eps):
    from theboss_gb300 import _native

    m, k = 15, 15
    U = _matrix(m, eps, 15)
    S, T = np.ones(m, dtype=np.int32), np.array([2, 2] + [1] * 10 + [0] * 3, dtype=np.int32)
    ref, tol = _glynn(U, list(range(k)), np.repeat(np.arange(m), T).tolist(), True)
    assert tol < 1e-4 * max(map(abs, ref))
    got = _native.submatrices_batch(U, S[None, :], T[None, :], _native.CHIN_HUH)[0]
    assert np.abs(got - np.array(ref)).max() <= tol, (eps, np.abs(got - np.array(ref)).max(), tol, np.abs(ref).max())


EXACT = [1e-3, 1e-6, 1e-9]


@pytest.mark.parametrize("eps", EXACT)
@pytest.mark.parametrize("k", [6, 11, 15])
def test_minors_of_exact_entries(k, eps):
    from theboss_gb300 import _native

    U = _exact_matrix(k, eps, k)
    T = np.array([2, 2] + [1] * (k - 5) + [0] * 3, dtype=np.int32)
    ref, tol = _glynn(U, list(range(k)), np.repeat(np.arange(k), T).tolist(), True, exact=True)
    got = _native.submatrices_batch(U, np.ones((1, k), dtype=np.int32), T[None, :], _native.CHIN_HUH)[0]
    assert np.abs(got - np.array(ref)).max() <= tol, (np.abs(got - np.array(ref)).max(), tol, np.abs(ref).max())


@pytest.mark.parametrize("eps", EXACT)
@pytest.mark.parametrize("S", [[1] * 8, [2, 2, 2, 2, 2, 1], [1] * 12], ids=["small", "multiple", "single"])
def test_permanents_of_exact_entries(S, eps):
    from theboss_gb300 import _native

    n = sum(S)
    U = _exact_matrix(n, eps, n)
    S = np.array(S + [0] * (n - len(S)), dtype=np.int32)
    T = np.array([2, 2] + [1] * (n - 4) + [0] * 2, dtype=np.int32)
    (ref,), tol = _glynn(U, np.repeat(np.arange(n), S).tolist(), np.repeat(np.arange(n), T).tolist(), False, exact=True)
    for count in (1, 40):
        got = _native.perm_batch(U, np.tile(S, (count, 1)), np.tile(T, (count, 1)), _native.CHIN_HUH)
        assert np.abs(got - ref).max() <= tol, (count, got[0], ref, tol)


@pytest.mark.parametrize("eps", EXACT)
def test_gradients_of_exact_entries(eps):
    from theboss_gb300 import _native

    n = 8
    U = _exact_matrix(n, eps, 80)
    # the sweep takes the inputs' digits: 2^2 3^3 / 2 codes against 2^8 / 2
    S, T = np.array([1, 1, 2, 2, 2, 0, 0, 0], dtype=np.int32), np.ones(n, dtype=np.int32)
    got = _native.perm_grad_batch(U, S[None, :], T[None, :])[1][0]
    cols = np.repeat(np.arange(n), S).tolist()
    for j in np.nonzero(T)[0]:  # d perm / d U[j, i] = T_j S_i minor(T - e_j, S - e_i)
        rows = np.repeat(np.arange(n), T - (np.arange(n) == j)).tolist()
        ref, tol = _glynn(U, cols, rows, True, exact=True)
        for i in np.nonzero(S)[0]:
            want = T[j] * sum(ref[q] for q in range(n) if cols[q] == i)
            assert abs(got[j, i] - want) <= T[j] * S[i] * tol, (j, i, got[j, i], want, tol)


@pytest.mark.parametrize("eps", EXACT)
def test_distributions_of_exact_entries(eps):
    from theboss_gb300 import _native

    n = 7
    U = _exact_matrix(n, eps, 70)
    S, T = np.ones(n, dtype=np.int32), np.array([2, 2] + [1] * (n - 4) + [0] * 2, dtype=np.int32)
    (ref,), tol = _glynn(U, list(range(n)), np.repeat(np.arange(n), T).tolist(), False, exact=True)
    got = _native.lossy_probabilities(U, S, T[None, :])[0] * 4.0
    assert abs(got - abs(ref) ** 2) <= 2.0 * abs(ref) * tol + tol ** 2 + 2.0 ** -50 * abs(ref) ** 2, (got, abs(ref) ** 2, tol)
