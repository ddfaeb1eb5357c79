"""The ticket range of an apply (mpdg_op_n_bricks): a stale counter anywhere in it leaves bricks to process, on meshes
whose launch cuts z into more or fewer parts than bricks of full height, and the handle recovers."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from tests.test_gpu_failure import SHORT

pytestmark = pytest.mark.gpu


def handle(kind, degree, cells):
    import torch

    from meltpooldg_b200.operators import AdvectionDiffusionOperator, HeatDiffuseOperator, Mesh, OlssonOperator

    mesh = Mesh(degree, cells, dirichlet_faces=63)
    if kind == "heat":
        return mesh, HeatDiffuseOperator(mesh, rho_cp=1.0, dt=1e-2, conductivity=1.0)
    if kind == "adv":
        return mesh, AdvectionDiffusionOperator(mesh, dt=1e-2, diffusivity=1e-3, velocity=[1.0] * 12)
    op = OlssonOperator(mesh, dt=1e-2, eps_normal=0.1, eps_tangential=0.1)
    op.set_normal(*[torch.ones(mesh.ndofs, dtype=torch.float64, device="cuda") for _ in range(3)])
    return mesh, op


# 96^3 at FE_Q(2): 576 segments of 12 layers against 864 bricks of 8; (64, 4, 8): 16 segments against 2 bricks
@pytest.mark.parametrize("kind,degree,cells", [("heat", 2, (96, 96, 96)), ("heat", 2, (64, 4, 8)), ("heat", 4, (64, 64, 64)),
                                               ("heat", 1, (160, 96, 70)), ("adv", 2, (96, 96, 96)), ("reinit", 2, (96, 96, 96))])
def test_every_ticket_in_the_range_is_useful(kind, degree, cells):
    import torch

    from meltpooldg_b200 import _lib as L

    mesh, op = handle(kind, degree, cells)
    lib = L.lib()
    n = lib.mpdg_op_n_bricks(op._h)
    assert n >= 1
    x = torch.tensor(uniform_dofs(mesh, seed=1), device="cuda")
    ref, y = torch.empty_like(x), torch.empty_like(x)
    op.vmult(ref, x)
    torch.cuda.synchronize()
    for ticket in sorted({1, n // 2, n - 1} - {0}):
        y.fill_(float("nan"))
        assert lib.mpdg_op_test_set_wait_limit(op._h, SHORT) == L.MPDG_OK
        assert lib.mpdg_op_test_set_ticket(op._h, ticket) == L.MPDG_OK
        op.vmult(y, x)
        torch.cuda.synchronize()
        assert op.device_errors() > 0
        # the bricks from the ticket on were processed
        assert torch.isfinite(y).any()
        assert lib.mpdg_op_test_set_wait_limit(op._h, 0) == L.MPDG_OK
        op.vmult(y, x)
        torch.cuda.synchronize()
        assert op.device_errors() == 0
        assert torch.max(torch.abs(y - ref)).item() <= 1e-13 * torch.max(torch.abs(ref)).item()
    assert np.isfinite(ref.sum().item())
