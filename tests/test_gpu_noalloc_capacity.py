"""The allocation-free entry point's fixed scratch (8 MiB): requests of the size that
the planners' rows, one 168-byte descriptor and one partial a thread (152 SMs) leave
room for are accepted, every variant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["RYSER", "CHIN_HUH", "GLYNN"])
@pytest.mark.parametrize("n,count", [(4, 18395), (8, 6061), (10, 4048), (12, 3021), (16, 1750), (20, 1136)])
def test_large_requests_fit(variant, n, count):
    import torch

    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    m, v = n + 2, getattr(_native, variant)
    U = haar_unitary(m, n)
    S = np.zeros((count, m), dtype=np.int32)
    S[:, :n] = 1
    T = np.roll(S, 1, axis=1).copy()
    out = torch.zeros(count, dtype=torch.complex128, device="cuda")
    _native.perm_batch_noalloc(U, S, T, v, out.data_ptr())
    torch.cuda.synchronize()
    ref = _native.perm_batch(U, S[:1], T[:1], v)[0]
    got = out.cpu().numpy()
    assert np.abs(got - ref).max() <= (1e-8 if variant == "RYSER" else 1e-12) * max(abs(ref), 1.0)


@pytest.mark.parametrize("sizes", [(4, 14), (14, 4), (0, 14)])
def test_mixed_requests(sizes):
    """Requests whose first permanent says little of the others: small ones first (the
    four-code rows of the rest do not fit), large ones first, empty ones first."""
    import torch

    from theboss_gb300 import _native
    from theboss_gb300.utilities import haar_unitary

    m, count = 16, 1000
    U = haar_unitary(m, 3)
    S = np.zeros((2 * count, m), dtype=np.int32)
    for h, n in enumerate(sizes):
        S[h * count:(h + 1) * count, :n] = 1
    T = np.roll(S, 2, axis=1).copy()
    out = torch.zeros(2 * count, dtype=torch.complex128, device="cuda")
    _native.perm_batch_noalloc(U, S, T, _native.GLYNN, out.data_ptr())
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for h in range(2):
        ref = _native.perm_batch(U, S[h * count:h * count + 1], T[h * count:h * count + 1], _native.GLYNN)[0]
        assert np.abs(got[h * count:(h + 1) * count] - ref).max() <= 1e-12 * max(abs(ref), 1.0)
