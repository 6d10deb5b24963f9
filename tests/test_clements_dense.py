"""The mesh as dense layers multiplied pairwise, whose derivatives clements_unitary
takes: the layers' own product, in another order; its value is that product's, to the
last bit; and nothing of a traced call stays behind (CPU)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


def _phases(m):
    g = torch.Generator().manual_seed(m)
    return [(torch.rand(m * (m - 1) // 2, generator=g, dtype=torch.float64) * 2 * np.pi).requires_grad_(True) for _ in "tp"]


@pytest.mark.parametrize("m", [1, 2, 3, 4, 7, 24])
def test_value(m):
    from theboss_gb300 import adjoint

    th, ph = _phases(m)
    loop = adjoint._layer_product(th, ph, m).detach()
    # m layers of two-term sums of numbers below 1, rounded at 2^-53 each, in two orders
    assert (adjoint._dense_product(th, ph, m).detach() - loop).abs().max() <= 4 * m * 2.0 ** -53
    assert torch.equal(adjoint.clements_unitary(th, ph).detach(), loop)


def test_after_a_traced_call():
    from torch._subclasses.fake_tensor import FakeTensor, FakeTensorMode

    from theboss_gb300 import adjoint

    m = 9  # no other test's
    with FakeTensorMode(allow_non_fake_inputs=True):
        adjoint.clements_unitary(*_phases(m))
    U = adjoint.clements_unitary(*_phases(m))
    assert not isinstance(U, FakeTensor)
    assert torch.equal(U.detach(), adjoint._layer_product(*_phases(m), m).detach())
