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
