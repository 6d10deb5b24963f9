"""Small permanents of submatrices far smaller than their rows' largest entries (weakly
coupled modes): every permanent keeps the precision of its own entries, alone and in
batches of one and of several passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [3, 40, 500])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 7])
def test_off_diagonal_permanents(n, count):
    from theboss_gb300 import _native

    m = 2 * n + 3
    rng = np.random.default_rng(n + count)
    G = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    U = np.eye(m) + 1e-9 * G  # inputs 0 .. n - 1, outputs among the other modes: no diagonal entry
    S = np.zeros((count, m), dtype=np.int32)
    S[:, :n] = 1
    T = np.zeros_like(S)
    for k in range(count):
        np.add.at(T[k], rng.integers(n, m, size=n), 1)
    small = 1e-9 * G  # the same submatrices, rounded differently: U's off-diagonal entries are these exactly
    got = _native.perm_batch(U, S, T, _native.GLYNN)
    for k in range(count):
        rows = np.repeat(np.arange(m), T[k])
        one = _native.perm_batch(np.ascontiguousarray(small[np.ix_(rows, np.arange(n))]), np.ones((1, n), np.int32),
                                 np.ones((1, n), np.int32), _native.GLYNN)[0]
        size = np.prod(np.abs(small[np.ix_(rows, np.arange(n))]).sum(axis=1))
        # at most 2^6 averaged products below size, each kept to 2^-52 and rounded at 2^-53 an addition
        assert abs(got[k] - one) <= 2.0 ** -44 * size, k
