"""Sweeps of so few codes that a thread takes fewer than eight (down to one): permanents
and all-minors permanents around the sizes where the share halves, against the sums
over a permanent's rows (Laplace expansion) and against batches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bunched", [0, 2])
@pytest.mark.parametrize("n", [2, 5, 9, 12, 15, 16, 17, 18])
def test_minors_expand_the_permanent(n, bunched):
    from theboss_gb300 import _native

    if bunched and n < 5:
        pytest.skip("too few modes")
    rng = np.random.default_rng(3 * n + bunched)
    m = n + 2
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    S = np.zeros((1, m), dtype=np.int32)
    S[0, :n] = 1
    for k in range(bunched):
        S[0, k] += 1
        S[0, n - 1 - k] -= 1
    T = np.zeros_like(S)
    np.add.at(T[0], rng.integers(0, m, size=n - 1), 1)
    o = int(rng.integers(0, m))
    T1 = T.copy()
    T1[0, o] += 1
    size = max(np.prod([(np.abs(U[j]) @ S[0]) ** t for j, t in enumerate(T1[0])]),
               np.prod([(np.abs(U[:, i]) @ T1[0]) ** s for i, s in enumerate(S[0])]))
    # terms below size, at most 2^19 of them (Ryser's and Chin-Huh's codes), each addition
    # rounded at 2^-53 of a partial sum; Ryser's terms are not averaged
    p = _native.perm_batch(U, S, T1, _native.GLYNN)[0]
    for variant, tol in ((_native.CHIN_HUH, 2.0 ** -42), (_native.RYSER, 2.0 ** (n - 41))):
        minors = _native.submatrices_batch(U, S, T, variant)[0]
        # column minors: perm(T + e_o) = sum_i S_i U[o, i] minor_i
        assert abs(np.sum(S[0] * U[o] * minors) - p) <= tol * size
