"""Column-marching heat apply at the edges of its tiling: one cell, one layer, partial columns in x and y, meshes
whose segment length differs (1 layer up to long segments with a shorter last one), rows that start at every
16-byte shift, vectors at every element offset, and each output mode, against the oracle."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from tests.gpu_util import rel_err, to_gpu
from tests.test_gpu_heat import heat_pair

pytestmark = pytest.mark.gpu

MESHES = [(1, 1, 1), (2, 1, 3), (31, 4, 2), (32, 5, 7), (33, 3, 1), (34, 9, 40), (65, 13, 19), (7, 101, 33)]


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("m", MESHES)
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_march_modes_and_offsets(degree, m, offset):
    import torch

    o, g, om, cm = heat_pair(degree, m, faces=0b011001, length=(1.1, 0.9, 1.3))
    x, b = uniform_dofs(om, seed=4), uniform_dofs(om, seed=5)
    ref = o.vmult(x)
    free = cm == 0

    def placed(v, dt):
        buf = torch.full((om.ndofs + offset,), float("nan"), dtype=dt, device="cuda")
        buf[offset:] = to_gpu(v, dt)
        return buf[offset:]

    # FP64 sums of at most 8 cells of 27 products each: 1e-12 as every FP64 apply here; FP32 2e-6
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-6)):
        y = placed(np.full(om.ndofs, np.nan), dt)
        g.vmult(y, placed(x, dt))
        assert rel_err(y.cpu().numpy(), ref) <= tol
    y = placed(b, torch.float64)
    g.vmult_add(y, placed(x, torch.float64), 0.5)
    assert rel_err(y.cpu().numpy(), b + 0.5 * np.where(free, ref, 0.0)) <= 1e-12
    r = placed(np.zeros(om.ndofs), torch.float64)
    g.residual(r, placed(b, torch.float64), placed(x, torch.float64))
    assert rel_err(r.cpu().numpy(), b - ref) <= 1e-12
    assert g.device_errors() == 0
