"""Advection apply (column-marching kernel) at the edges of its tiling: partial columns, one cell, several segments,
Dirichlet faces with and without per-DoF flags, rows at every 16-byte shift and vectors at every element offset,
each output mode, against the oracle."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from oracle.oracle import Operator as OOp
from tests.gpu_util import meshes, rel_err, to_gpu

pytestmark = pytest.mark.gpu

VEL = [0.5, -0.5, 0.1, 0.0, -1.0, 0.2, 1.0, 0.0, 0.0, 0.3, 0.0, -0.2]
DT, THETA, EPS = 5e-3, 0.7, 2e-3


def operator(degree, m, faces, mask=None, theta=THETA):
    from meltpooldg_b200.operators import AdvectionDiffusionOperator

    om, gm, cm = meshes(degree, m, faces=faces, mask=mask, length=(1.0, 0.9, 1.2))
    return om, cm, AdvectionDiffusionOperator(gm, dt=DT, theta=theta, diffusivity=EPS, velocity=VEL)


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("m", [(1, 1, 1), (33, 2, 3), (7, 9, 2), (40, 5, 13)])
@pytest.mark.parametrize("masked", [False, True])
def test_advection_modes(degree, m, masked):
    import torch

    rng = np.random.default_rng(7)
    n = np.prod([degree * c + 1 for c in m])
    mask = (rng.random(n) < 0.2).astype(np.uint8) if masked else None
    om, cm, g = operator(degree, m, 0b100010, mask)
    x, b = uniform_dofs(om, seed=1), uniform_dofs(om, seed=2)
    ref = OOp(om, "advdiff", cmask=cm, dt=DT, theta=THETA, eps=EPS, vel=VEL).vmult(x)
    for offset in (0, 1, 2, 3):
        for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-6)):
            xs = torch.full((om.ndofs + offset,), float("nan"), dtype=dt, device="cuda")
            ys = torch.full_like(xs, float("nan"))
            xs[offset:] = to_gpu(x, dt)
            g.vmult(ys[offset:], xs[offset:])
            assert rel_err(ys[offset:].cpu().numpy(), ref) <= tol
    y = to_gpu(b)
    g.vmult_add(y, to_gpu(x), -0.5)
    assert rel_err(y.cpu().numpy(), b - 0.5 * np.where(cm == 0, ref, 0.0)) <= 1e-12
    r = to_gpu(np.zeros(om.ndofs))
    g.residual(r, to_gpu(b), to_gpu(x))
    assert rel_err(r.cpu().numpy(), b - ref) <= 1e-12
    assert g.device_errors() == 0
