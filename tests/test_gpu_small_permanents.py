"""Small permanents (at most 10 particles): the split of a permanent's sign vectors
over 1 to 128 lanes (by the count), the host-gathered form of a few and the general
one, and the rows that have no fixed-point scale (sizes near the ends of the
exponent range, infinities, NaN), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 13


def _matrix(seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(M, M)) + 1j * rng.normal(size=(M, M))


def _patterns(rng, n, count):
    S = np.zeros((count, M), dtype=np.int32)
    T = np.zeros((count, M), dtype=np.int32)
    for k in range(count):
        np.add.at(S[k], rng.integers(0, M, size=n), 1)
        np.add.at(T[k], rng.integers(0, M, size=n), 1)
    return S, T


def _largest(U, S, T):
    """No term of the Glynn sum exceeds it: prod over the output particles of sum_i S_i |U|."""
    A = np.abs(U) @ S
    return float(np.prod([A[j] ** t for j, t in enumerate(T)]))


# each of the 2^(L-1) terms is within L 2^-56 + 2^-53 of the largest, their FP64 sum adds 2^-53 a term
TOL = 2.0 ** -43


@pytest.mark.parametrize("count", [1, 3, 16, 17, 300, 40000])
def test_lanes_per_permanent(oracle, count):
    from theboss_gb300 import _native

    rng = np.random.default_rng(count)
    U = _matrix(count)
    S, T = (np.concatenate(x) for x in zip(*[_patterns(rng, n, max(1, count // 10)) for n in range(1, 11)]))
    S, T = S[:max(count, 1)] if count < 10 else S, T[:max(count, 1)] if count < 10 else T
    got = _native.perm_batch(U, S, T, _native.CHIN_HUH)
    for k in rng.choice(len(S), size=min(len(S), 60), replace=False):
        ref = oracle.perm(U, S[k].tolist(), T[k].tolist())
        assert abs(got[k] - ref) <= TOL * _largest(U, S[k], T[k]), (k, S[k], T[k], got[k], ref)


@pytest.mark.parametrize("n", [1, 2, 5, 9, 10])
def test_single_of_every_size(oracle, n):
    from theboss_gb300 import _native

    rng = np.random.default_rng(50 + n)
    U = _matrix(n)
    S, T = _patterns(rng, n, 1)
    got = _native.perm_batch(U, S, T, _native.RYSER)[0]
    ref = oracle.perm(U, S[0].tolist(), T[0].tolist())
    assert abs(got - ref) <= TOL * _largest(U, S[0], T[0])


@pytest.mark.parametrize("count", [1, 200])
@pytest.mark.parametrize("kind", ["tiny", "huge", "inf", "nan"])
def test_rows_without_a_fixed_point_scale(oracle, kind, count):
    from theboss_gb300 import _native

    rng = np.random.default_rng(7)
    U = _matrix(9)
    U[4] *= {"tiny": 1e-280, "huge": 1e280, "inf": 1.0, "nan": 1.0}[kind]
    if kind in ("inf", "nan"):
        U[4, 2] = np.inf if kind == "inf" else np.nan
    S = np.zeros((count, M), dtype=np.int32)
    S[:, [0, 1, 2, 3]] = 1
    T = np.zeros((count, M), dtype=np.int32)
    T[:, [3, 4, 5, 6]] = 1
    if count > 1:
        T[1:, 4], T[1:, 7] = 0, 1  # the others do not touch the row
    got = _native.perm_batch(U, S, T, _native.GLYNN)
    if kind in ("inf", "nan"):
        assert not np.isfinite(got[0])
    else:
        ref = oracle.perm(U, S[0].tolist(), T[0].tolist())
        assert abs(got[0] - ref) <= TOL * _largest(U, S[0], T[0])
    if count > 1:
        ref = oracle.perm(U, S[1].tolist(), T[1].tolist())
        assert np.all(np.abs(got[1:] - ref) <= TOL * _largest(U, S[1], T[1]))
