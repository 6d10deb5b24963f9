"""The integer-pipe product chains of the sweeps (permanents, all-minors) at every
kind of factor count: one to three factors (a single chain or none), the first
split into two chains, odd splits, the register steps at 16/17 and the largest.
The input side is a few multiply occupied modes, so that the codes are few and the
oracle (Glynn's sum in exact rational arithmetic) stays cheap at 32 factors."""
import itertools
from fractions import Fraction
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 4, 5, 8, 15, 16, 17, 24, 31, 32]


def _cmul(a, b):
    return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]


def _glynn(U, S, rows, weights=None):
    """(sum over codes of sign ΠC [w] Π_f s_f as exact rationals, the same of absolute
    values in float) times 2^-n; rows: the factors' output modes."""
    modes = [i for i, s in enumerate(S) if s]
    n = sum(S)
    tot = (Fraction(0), Fraction(0))
    l1 = 0.0
    for r in itertools.product(*[range(S[i] + 1) for i in modes]):
        p = (Fraction(1), Fraction(0))
        mag = 1.0
        for f in rows:
            s = (Fraction(0), Fraction(0))
            for i, ri in zip(modes, r):
                k = S[i] - 2 * ri
                s = s[0] + k * Fraction(U[f, i].real), s[1] + k * Fraction(U[f, i].imag)
            p = _cmul(p, s)
            mag *= abs(complex(float(s[0]), float(s[1])))
        c = 1
        for i, ri in zip(modes, r):
            c *= comb(S[i], ri)
        w = 1 if weights is None else weights(r, modes)
        sg = -c * w if sum(r) % 2 else c * w
        tot = tot[0] + sg * p[0], tot[1] + sg * p[1]
        l1 += c * abs(w) * mag
    return complex(float(tot[0] / 2 ** n), float(tot[1] / 2 ** n)), l1 / 2.0 ** n


def _case(nf, seed):
    rng = np.random.default_rng(seed)
    m = nf + 3
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    U *= (2.0 ** -rng.integers(0, 12, size=m))[:, None]  # rows of different sizes: every factor its own scale
    return U


def _split(n):
    """n particles over up to four modes, one or two of them single."""
    if n < 4:
        return [1] * n
    return [1, 1, (n - 2) // 2, n - 2 - (n - 2) // 2]


def _tolerance(U, S, rows, l1):
    # a product is off by less than 2^-56 of (the chain so far) x (the factor's largest possible sum), the
    # entries are rounded to 2^-61 of it, and the FP64 additions by 2^-53 each of at most their L1 sum
    B = np.prod([sum(s * max(abs(U[f, i].real), abs(U[f, i].imag)) for i, s in enumerate(S)) * np.sqrt(2.0)
                 for f in rows])
    return len(rows) * 2.0 ** -54 * B + 2.0 ** -44 * l1


@pytest.mark.parametrize("nf", COUNTS)
def test_permanent_chains(nf):
    from theboss_gb300 import _native

    U = _case(nf, nf)
    m = U.shape[0]
    S = np.array((_split(nf) + [0] * m)[:m], dtype=np.int32)
    T = np.zeros(m, dtype=np.int32)
    T[m - nf:] = 1
    rows = list(range(m - nf, m))
    ref, l1 = _glynn(U, S.tolist(), rows)
    got = _native.perm_bench(U, S[None, :], T[None, :], _native.CHIN_HUH, 0, 1, 0)["results"][0]
    assert abs(got - ref) <= _tolerance(U, S, rows, l1), (nf, got, ref)


@pytest.mark.parametrize("nf", COUNTS)
def test_minors_chains(nf):
    from theboss_gb300 import _native

    U = _case(nf, 100 + nf)
    m = U.shape[0]
    k = min(nf + 1, 32)  # the input's particles; 32 factors have 32 input particles' minors as rectangular sums
    S = np.array((_split(k) + [0] * m)[:m], dtype=np.int32)
    T = np.zeros(m, dtype=np.int32)
    T[m - nf:] = 1
    rows = list(range(m - nf, m))
    got = _native.submatrices_batch(U, S[None, :], T[None, :], _native.CHIN_HUH)[0]
    for i in np.nonzero(S)[0]:
        # S_i minor_i = 2^-k sum_r sign ΠC (S_i - 2 r_i) Π_f s_f
        ref, l1 = _glynn(U, S.tolist(), rows, lambda r, modes: int(S[i]) - 2 * r[modes.index(i)])
        tol = _tolerance(U, S, rows, l1) * int(S[i])
        assert abs(got[i] * int(S[i]) - ref) <= tol, (nf, i, got[i], ref)
