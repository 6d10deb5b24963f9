"""Sweep rows made on the GPU (batches) against rows made on the host (one permanent
a call): the same permanents for every formula, odd and even factor counts, doubly
and triply occupied modes on either side and both orientations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _states(rng, m, n, count, most):
    out = np.zeros((count, m), dtype=np.int32)
    for k in range(count):
        while out[k].sum() < n:
            i = int(rng.integers(0, m))
            if out[k, i] < most:
                out[k, i] += 1
    return out


def _case(n, most):
    rng = np.random.default_rng(10 * n + most)
    m = n + 2
    U = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    U *= (2.0 ** -rng.integers(0, 8, size=m))[:, None]
    S, T = _states(rng, m, n, 6, most), _states(rng, m, n, 6, 4 - most)
    size = [np.prod([(np.abs(U[j]) @ s) ** t for j, t in enumerate(tt)]) for s, tt in zip(S, T)]
    return U, S, T, np.array(size, dtype=float)


@pytest.mark.parametrize("most", [1, 2, 3])
@pytest.mark.parametrize("n", [11, 12, 13, 16])
@pytest.mark.parametrize("variant", ["RYSER", "CHIN_HUH", "GLYNN"])
def test_batches_equal_single_calls(variant, n, most):
    from theboss_gb300 import _native

    U, S, T, size = _case(n, most)
    v = getattr(_native, variant)
    got = _native.perm_batch(U, S, T, v)
    for k in range(len(S)):
        one = _native.perm_batch(U, S[k:k + 1], T[k:k + 1], v)[0]
        # the sums of at most 2^16 terms below size 2^n (Ryser; Glynn's average is below size), in two
        # orders, each addition rounded at 2^-53 of its partial sum
        tol = size[k] * (2.0 ** (n - 42) if variant == "RYSER" else 2.0 ** -42)
        assert abs(got[k] - one) <= tol, (k, got[k], one)
