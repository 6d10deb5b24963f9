"""The four-code kernels (permanents, all-minors) against Glynn's sum in exact integers at
every kind of factor count: odd last factors, partial rounds of pairs, up to 16 pairs;
four single modes (two low digits, one outer, one held) and two multiply occupied ones, so
that the codes are few."""
import itertools
from fractions import Fraction
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BITS = 120  # the entries are multiples of 2^-120


def _case(nf, seed):
    rng = np.random.default_rng(seed)
    m = nf + 3
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    return U * (2.0 ** -rng.integers(0, 12, size=m))[:, None]  # rows of different sizes: every factor its own scale


def _split(n):
    return [1] * n if n < 8 else [1, 1, 1, 1, (n - 4) // 2, n - 4 - (n - 4) // 2]


def _int(x):
    v = Fraction(float(x)) * 2 ** BITS
    assert v.denominator == 1
    return v.numerator


def _glynn(U, S, rows):
    """The permanent's sum, the weighted ones (S_i minor_i) and the bound on their error."""
    modes = [i for i, s in enumerate(S) if s]
    n = sum(S)
    E = [[(_int(U[r, i].real), _int(U[r, i].imag)) for i in modes] for r in rows]
    F = U[np.ix_(rows, modes)]
    mult = np.array([S[i] for i in modes])
    # the entries' roundings: half a unit each, 2^-61 of the factor's largest possible sum at most
    delta = n * np.sqrt(0.5) * 2.0 ** -61 * (np.maximum(abs(F.real), abs(F.imag)) * mult).sum(axis=1)
    out = [[0, 0] for _ in range(1 + len(modes))]
    tol = 0.0
    for r in itertools.product(*[range(S[i] + 1) for i in modes]):
        d = [S[i] - 2 * ri for i, ri in zip(modes, r)]
        p, mag, wide = (1, 0), 1.0, 1.0
        for row, de in zip(E, delta):
            s = (sum(x * k[0] for x, k in zip(d, row)), sum(x * k[1] for x, k in zip(d, row)))
            p = p[0] * s[0] - p[1] * s[1], p[0] * s[1] + p[1] * s[0]
            a = abs(complex(s[0] / 2 ** BITS, s[1] / 2 ** BITS))
            mag *= a
            wide *= a + de
        c = 1
        for i, ri in zip(modes, r):
            c *= comb(S[i], ri)
        for k, w in enumerate([1] + d):
            sg = -c * w if sum(r) % 2 else c * w
            out[k][0] += sg * p[0]
            out[k][1] += sg * p[1]
        # every product 2^-54 of its size per factor, and the FP64 additions (at most 2^6 in a row)
        tol += c * (wide - mag + (len(rows) * 2.0 ** -54 + 2.0 ** -47) * wide)
    unit = 2 ** (BITS * len(rows) + n)
    vals = [complex(Fraction(re, unit), Fraction(im, unit)) for re, im in out]
    return vals[0], dict(zip(modes, vals[1:])), tol / 2.0 ** n


@pytest.mark.parametrize("nf", [3, 4, 5, 6, 7, 8, 15, 16, 17, 23, 24, 31, 32])
def test_permanents(nf):
    from theboss_gb300 import _native

    U = _case(nf, nf)
    m = U.shape[0]
    S = np.array(_split(nf) + [0] * (m - len(_split(nf))), dtype=np.int32)
    T = np.array([0] * 3 + [1] * nf, dtype=np.int32)
    ref, _, tol = _glynn(U, S.tolist(), list(range(3, m)))
    got = _native.perm_bench(U, S[None, :], T[None, :], _native.CHIN_HUH, 0, 1, 0)["results"][0]
    assert abs(got - ref) <= tol, (nf, got, ref, tol)


@pytest.mark.parametrize("nf", [14, 15, 16, 17, 20, 23, 24, 30, 31])
def test_minors(nf):
    from theboss_gb300 import _native

    U = _case(nf, 100 + nf)
    m, k = U.shape[0], nf + 1
    S = np.array(_split(k) + [0] * (m - len(_split(k))), dtype=np.int32)
    T = np.array([0] * 3 + [1] * nf, dtype=np.int32)
    _, ref, tol = _glynn(U, S.tolist(), list(range(3, m)))
    got = _native.submatrices_batch(U, S[None, :], T[None, :], _native.CHIN_HUH)[0]
    for i, v in ref.items():
        assert abs(got[i] * int(S[i]) - v) <= int(S[i]) * tol, (nf, i, got[i], v, tol)
