"""The mesh's two forms (dense layers multiplied pairwise, and layer by layer): the
same unitary and the same phase gradients, at the sizes where the pairwise product
ends on an odd layer or has one layer only (CPU)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m", [1, 2, 3, 4, 7, 24])
def test_dense_layers_equal_the_loop(m, monkeypatch):
    from theboss_gb300 import adjoint

    p = m * (m - 1) // 2
    g = torch.Generator().manual_seed(m)
    th = (torch.rand(p, generator=g, dtype=torch.float64) * 2 * np.pi).requires_grad_(True)
    ph = (torch.rand(p, generator=g, dtype=torch.float64) * 2 * np.pi).requires_grad_(True)
    w = torch.randn(m, m, generator=g, dtype=torch.complex128)

    def value_and_grad():
        U = adjoint.clements_unitary(th, ph)
        s = (U * w).real.sum()
        return U.detach(), torch.autograd.grad(s, [th, ph]) if p else ()

    U, dU = value_and_grad()
    monkeypatch.setattr(adjoint, "_DENSE_LAYERS", 0)
    V, dV = value_and_grad()
    # m layers of two-term sums of numbers below 1, rounded at 2^-53 each, in two orders
    tol = 4 * m * 2.0 ** -53
    assert (U - V).abs().max() <= tol
    for a, b in zip(dU, dV):
        assert (a - b).abs().max() <= tol * float(w.abs().sum())
