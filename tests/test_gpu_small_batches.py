"""Batches of small permanents of mixed particle counts (modes decoded and rows scaled on
the GPU) against the same permanents one by one (both done on the host)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [17, 40, 333])
@pytest.mark.parametrize("m, width", [(1, 1), (5, 5), (33, 31), (70, 64)])
def test_mixed_counts(m, width, count):
    from theboss_gb300 import _native

    rng = np.random.default_rng(m + count)
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    S = np.zeros((count, width), dtype=np.int32)
    T = np.zeros_like(S)
    for k in range(count):
        n = int(rng.integers(0, 11))
        np.add.at(S[k], rng.integers(0, width, size=n), 1)
        np.add.at(T[k], rng.integers(0, width, size=n), 1)
    got = _native.perm_batch(U, S, T, _native.GLYNN)
    for k in range(count):
        one = _native.perm_batch(U, S[k:k + 1], T[k:k + 1], _native.GLYNN)[0]
        size = np.prod([(np.abs(U[j, :width]) @ S[k]) ** t for j, t in enumerate(T[k])])
        # at most 2^9 averaged products below size; the two scale rows by different powers of two:
        # entries rounded at 2^-60 of their row's bound, products kept to 2^-52, sums to 2^-53 each
        assert abs(got[k] - one) <= 2.0 ** -43 * size, k
