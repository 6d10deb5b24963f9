"""Levels whose samples have different code counts (bunched inputs): a batch's samples
equal those of the same stream taken one at a time, whose levels have one code count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 6, 40])
@pytest.mark.parametrize("n, bunched", [(10, 1), (13, 3), (17, 2), (19, 1)])
def test_batch_equals_single_samples(n, bunched, count):
    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    m = n + 6
    S = np.zeros(m, dtype=np.int32)
    S[:n] = 1
    for k in range(bunched):
        S[k] += 1
        S[n - 1 - k] -= 1
    U = haar_unitary(m, n)
    np.random.seed(n + count)
    batch = _native.gccb_sample(U, S, None, count)
    for k in range(count):
        np.random.seed(n + count)
        one = _native.gccb_sample_slice(U, S, None, count, k, 1)
        np.testing.assert_array_equal(batch[k], one[0])
