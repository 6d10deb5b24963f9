"""Gradients whose walkers are summed in parts (one or a few permanents), with rows made
on the host (fewer than 4 permanents) and on the GPU: every output
mode's row is homogeneous in the permanent, sum_i U[j, i] dP/dU[j, i] = T_j P, and the
permanent is the batched permanents'.  Sizes around the first split and the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 5])
@pytest.mark.parametrize("bunched", [0, 2])
@pytest.mark.parametrize("n", [10, 11, 12, 13, 15, 18])
def test_rows_are_homogeneous(n, bunched, count):
    from theboss_gb300 import _native

    rng = np.random.default_rng(100 * n + 10 * bunched + count)
    m = n + 3
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    S = np.zeros((count, m), dtype=np.int32)
    S[:, :n] = 1
    for k in range(bunched):
        S[:, k] += 1
        S[:, n - 1 - k] -= 1
    T = np.zeros_like(S)
    for k in range(count):
        np.add.at(T[k], rng.integers(0, m, size=n), 1)
    perms, grads = _native.perm_grad_batch(U, S, T)
    ref = _native.perm_batch(U, S, T, _native.GLYNN)
    for k in range(count):
        # the largest product a sweep over the input modes' or the output modes' codes can meet
        size = max(np.prod([(np.abs(U[j]) @ S[k]) ** t for j, t in enumerate(T[k])]),
                   np.prod([(np.abs(U[:, i]) @ T[k]) ** s for i, s in enumerate(S[k])]))
        # sums of at most 2^17 products below size (their average is returned), each kept to 2^-52 of
        # its size, in orders that lose at most 2^-53 an addition of partial sums below size
        tol = 2.0 ** -42 * size
        assert abs(perms[k] - ref[k]) <= tol
        g = grads[k].reshape(m, m)
        for j in range(m):
            # an entry's products leave out one factor: size over that factor's bound; entries i of
            # row j are off by at most 2^-42 of that each
            loo = size / min([np.abs(U[q]) @ S[k] for q in range(m) if T[k, q]] +
                             [np.abs(U[:, i]) @ T[k] for i in range(m) if S[k, i]])
            off = 2.0 ** -42 * loo * n * n * np.abs(U[j]).sum()
            assert abs(np.sum(U[j] * g[j]) - T[k, j] * perms[k]) <= off + tol * T[k, j], (k, j)
