"""The sampler's first levels in one launch: samples equal to those of the float-pair
arithmetic, whose levels are launched one by one, at and beside the last level of the
launch, for one and several outputs a lane, bunched inputs and losses."""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _samples(U, S, weights, count, seed):
    from theboss_gb300 import _native

    np.random.seed(seed)
    return _native.gccb_sample(U, S, weights, count)


@pytest.mark.parametrize("count", [1, 6, 300])
@pytest.mark.parametrize("bunched", [0, 1, 3])
@pytest.mark.parametrize("eta", [1.0, 0.6])
@pytest.mark.parametrize("n, m", [(1, 1), (2, 40), (7, 16), (8, 33), (9, 64), (11, 256)])
def test_samples_do_not_depend_on_the_launches(n, m, eta, bunched, count):
    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    S = np.zeros(m, dtype=np.int32)
    S[:n] = 1
    for k in range(min(bunched, n // 2)):
        S[k] += 1
        S[n - 1 - k] -= 1
    U = haar_unitary(m, 10 * n + m)
    weights = None if eta == 1.0 else [comb(n, l) * eta ** l * (1 - eta) ** (n - l) for l in range(n + 1)]
    got = _samples(U, S, weights, count, n + count)
    before = _native.minors_arithmetic()
    try:
        _native.minors_arithmetic(0)
        levels = _samples(U, S, weights, count, n + count)
    finally:
        _native.minors_arithmetic(before)
    # integers: a draw is decided exactly, by the sequential rule where a cdf step is near
    np.testing.assert_array_equal(got, levels)
    if eta == 1.0:
        assert (got.sum(axis=1) == n).all()
