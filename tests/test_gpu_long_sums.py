"""Sums of many codes a lane: a diagonal matrix, whose signed products all equal the
permanent, so that the rounding of a sum taken in one piece adds up in one direction."""
from fractions import Fraction
from math import prod

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_equal_terms():
    from theboss_gb300 import _native

    n, m, count = 26, 30, 64
    rng = np.random.default_rng(26)
    u = rng.uniform(0.5, 1.0, size=m)
    S = np.zeros((count, m), dtype=np.int32)
    for k in range(count):
        S[k, rng.choice(m, size=n, replace=False)] = 1
    ref = np.array([float(prod(Fraction(u[i]) for i in np.nonzero(s)[0])) for s in S])
    got = _native.perm_batch(np.diag(u).astype(complex), S, S, _native.GLYNN)
    # steps of four codes a walker: 2^23 a permanent over at least 152 * 32 walkers for all 64, in sums of
    # 64 steps, summed; then 32 lanes and the groups' partials (256 threads); every addition 2^-53 of at most
    # the (positive) total; the product n 2^-55
    steps = 64 * 2.0 ** 23 / (152 * 32 * 3)
    groups = 152 * 32 * 3 / 64 / 8 / 256
    bound = (64 + steps / 64 + 5 + groups + 8) * 2.0 ** -53 + n * 2.0 ** -55
    err = np.abs(got - ref) / ref
    assert err.max() <= bound, (err.max(), bound)
