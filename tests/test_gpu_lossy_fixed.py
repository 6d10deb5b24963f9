"""Exact distributions with row sums and products in fixed and block floating point
against the FP64 kernels, which a matrix with an entry beyond every scale takes: the
particle counts around the step to several blocks of sign vectors, and the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, m", [(1, 3), (2, 4), (4, 5), (5, 5), (6, 5), (7, 4), (10, 4)])
def test_fixed_equals_fp64(n, m):
    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary, possible_states_array

    U = haar_unitary(m, n)
    U[0, 0] = 0.0
    V = U.copy()
    V[0, 0] = 1e-290  # changes no result by more than 1e-289, and has no scale
    S = np.zeros(m, dtype=np.int32)
    for k in range(n):
        S[k % m] += 1
    outs = np.concatenate([possible_states_array(l, m) for l in range(n + 1)]).astype(np.int32)
    p = _native.lossy_probabilities(U, S, outs)
    q = _native.lossy_probabilities(V, S, outs)
    # |perm|^2 <= size^2 with size = prod of the rows' 1-norms, summed over the lossy inputs and
    # divided; both kernels keep a permanent to 2^-45 of size (512 sums, 10 products in FP64)
    norms = np.abs(U).sum(axis=1)
    for l in range(n + 1):
        size = np.maximum(norms.max(), 1.0) ** l
        mine = outs.sum(axis=1) == l
        assert np.abs(p[mine] - q[mine]).max() <= 2.0 ** -43 * size ** 2
    assert np.isfinite(p).all()
