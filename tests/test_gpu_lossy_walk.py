"""The walked distribution kernels: particle counts on both sides of the step from
several inputs per warp to several blocks of sign vectors per input (5, 6, 7, 8),
outcomes in any order (shared prefixes of every length, repeats, all counts mixed),
chunk remainders, and inputs with doubly occupied modes, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _outcomes(rng, m, ls, order):
    T = np.zeros((len(ls), m), dtype=np.int32)
    for k, l in enumerate(ls):
        np.add.at(T[k], rng.integers(0, m, size=l), 1)
    if order == "sorted":  # by count, then descending lexicographic, as the calculators list them
        keys = [(int(t.sum()), tuple(-t)) for t in T]
        T = T[sorted(range(len(ls)), key=lambda k: keys[k])]
    elif order == "repeated":
        T = np.repeat(T, 2, axis=0)
    return T


@pytest.mark.parametrize("order", ["random", "sorted", "repeated"])
@pytest.mark.parametrize("S,count", [([1, 1, 1, 0, 0], 9), ([1] * 6 + [0] * 3, 130), ([2, 1, 1, 2, 1, 0, 1, 0], 150),
                                     ([1] * 8 + [0] * 2, 70)])
def test_outcomes_in_any_order(oracle, S, count, order):
    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    m, n = len(S), sum(S)
    rng = np.random.default_rng(count)
    U = haar_unitary(m, count)
    T = _outcomes(rng, m, rng.integers(0, n + 1, size=count), order)
    got = _native.lossy_probabilities(U, S, T)
    for k in rng.choice(len(T), size=min(len(T), 40), replace=False):
        l = int(T[k].sum())
        ref = 1.0 if l == 0 else oracle.fixed_loss_probability(U, S, T[k].tolist())
        # squares of sums of at most 2^(l-1) products of l row sums below sqrt(l), rounded at 2^-53 an
        # operation: 2^-43 of 1 covers them at l = 8
        assert abs(got[k] - ref) <= 2.0 ** -43 * max(abs(ref), 1e-3), (T[k], got[k], ref)
