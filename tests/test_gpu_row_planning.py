"""Batches on both sides of the rule that has their rows made on the GPU or on the host
(few permanents in many modes: the host): the same permanents and gradients as one by
one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,count", [(24, 4), (24, 8), (200, 8), (200, 40), (512, 4)])
def test_batches_equal_single_calls(m, count):
    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    n = 12
    rng = np.random.default_rng(m + count)
    U = haar_unitary(m, m)
    S, T = np.zeros((2, count, m), dtype=np.int32)
    for k in range(count):
        S[k, rng.choice(m, size=n, replace=False)] = 1
        T[k, rng.choice(m, size=n, replace=False)] = 1
    # every sum has 2^11 terms below size (the larger of the two orientations' products of 1-norms);
    # the additions, 2^-53 of a partial sum each, differ in their order only
    A = np.abs(U)
    size = np.array([max(np.prod((A @ s)[t > 0]), np.prod((A.T @ t)[s > 0])) for s, t in zip(S, T)])
    got = _native.perm_batch(U, S, T, _native.GLYNN)
    _, grads = _native.perm_grad_batch(U, S, T)
    for k in range(count):
        assert abs(got[k] - _native.perm_batch(U, S[k:k + 1], T[k:k + 1], _native.GLYNN)[0]) <= size[k] * 2.0 ** -42
        one = _native.perm_grad_batch(U, S[k:k + 1], T[k:k + 1])[1][0]
        # a derivative's terms lack one factor: below size over the smallest 1-norm
        least = min((A @ S[k])[T[k] > 0].min(), (A.T @ T[k])[S[k] > 0].min())
        assert np.abs(grads[k] - one).max() <= size[k] / least * 2.0 ** -42
