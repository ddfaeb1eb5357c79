"""Narrow band at the threshold: a Gauss point whose level set differs from it by rounding alone belongs to the
banded apply and to its diagonal alike."""
import numpy as np
import pytest

from tests.gpu_util import to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 2, 3])
def test_apply_and_diagonal_agree_at_the_threshold(degree):
    import torch

    from meltpooldg_b200.operators import HeatDiffuseOperator, Mesh

    mesh = Mesh(degree, (2, 1, 1))
    op = HeatDiffuseOperator(mesh, rho_cp=1.0, dt=1.0, conductivity=0.1)
    x, y = torch.zeros(mesh.ndofs, dtype=torch.float64, device="cuda"), torch.empty(mesh.ndofs, dtype=torch.float64, device="cuda")
    inv = torch.empty_like(x)
    for level in np.random.default_rng(1).uniform(0.5, 2.0, 20):
        # a constant level set at the threshold: interpolated, it lies on either side of it by rounding
        ls = to_gpu(np.full(mesh.ndofs, level))
        op.set_narrow_band(ls, float(level))
        op.compute_inverse_diagonal_from_matrixfree(inv)
        apply = np.empty(mesh.ndofs)
        for i in range(mesh.ndofs):
            x.zero_()
            x[i] = 1.0
            op.vmult(y, x)
            apply[i] = y[i].item()
        # entries without a point in the band have the inverse 1
        expect = np.where(apply > 1e-14, 1.0 / np.where(apply > 1e-14, apply, 1.0), 1.0)
        # sums of at most 2 cells of 64 points
        assert np.max(np.abs(inv.cpu().numpy() / expect - 1.0)) <= 1e-12, level
    assert op.device_errors() == 0
