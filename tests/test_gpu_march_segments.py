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


@pytest.mark.parametrize("degree", [3, 4])
@pytest.mark.parametrize("m", [(1, 1, 1), (5, 6, 9), (33, 3, 5), (64, 2, 17), (32, 1, 40)])
def test_pencil_parts(degree, m):
    """Pencil apply on meshes whose z direction is cut into few, many and unequal parts."""
    import torch

    o, g, om, cm = heat_pair(degree, m, faces=0b100110, length=(1.1, 0.9, 1.3))
    x, b = uniform_dofs(om, seed=6), uniform_dofs(om, seed=7)
    ref = o.vmult(x)
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-6)):
        y = torch.full((om.ndofs,), float("nan"), dtype=dt, device="cuda")
        g.vmult(y, to_gpu(x, dt))
        assert rel_err(y.cpu().numpy(), ref) <= tol
    y = to_gpu(b)
    g.vmult_add(y, to_gpu(x), 2.0)
    assert rel_err(y.cpu().numpy(), b + 2.0 * np.where(cm == 0, ref, 0.0)) <= 1e-12
    assert g.device_errors() == 0


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("m", [(1, 2, 1), (33, 5, 3), (40, 9, 11)])
@pytest.mark.parametrize("parts", ["all", "no_q", "no_old", "only_T"])
def test_rhs_in_one_pass(degree, m, parts):
    """create_rhs accumulates M (rho c_p / dt (T_old - T) + q) - K T, for each optional input left out."""
    o, g, om, cm = heat_pair(degree, m, faces=0b010100, length=(1.1, 0.9, 1.3))
    T, old, q, dst = (uniform_dofs(om, seed=s) for s in (1, 2, 3, 4))
    old = None if parts in ("no_old", "only_T") else old
    q = None if parts in ("no_q", "only_T") else q
    y = to_gpu(dst)
    g.create_rhs(y, to_gpu(T), None if old is None else to_gpu(old), None if q is None else to_gpu(q))
    zero = np.zeros(om.ndofs)
    # T_old left out drops its term (not the one of T), as a zero vector does
    ref = dst.copy()
    o.create_rhs(ref, T, zero if old is None else old, zero if q is None else q)
    # sums of two products of 27 terms with coefficients up to rho c_p / dt = 130
    assert rel_err(y.cpu().numpy(), ref) <= 1e-12
    assert g.device_errors() == 0
