"""Reinitialisation, projections and temperature-dependent material (column-marching kernels that zero constrained
values in the staged rows) at the edges of their tiling: one cell, partial and full columns in x and y, a cell beyond
a column, several segments, Dirichlet faces with and without per-DoF flags inside the mesh, vectors at every element
offset and each output mode, against the oracles."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from oracle import reinit as oracle_reinit
from oracle import solidification as oracle_solid
from tests.gpu_util import meshes, rel_err, to_gpu

pytestmark = pytest.mark.gpu

MESHES = [(1, (1, 1, 1)), (1, (33, 5, 3)), (1, (65, 4, 2)), (1, (40, 9, 11)), (2, (1, 1, 1)), (2, (33, 5, 3)), (2, (32, 8, 5)),
          (2, (40, 9, 11)), (3, (1, 1, 1)), (3, (33, 5, 3)), (3, (34, 4, 2)),
          # columns of 16 x 8 cells: one and several, partial in x and y
          (1, (8, 17, 30)), (2, (5, 9, 6)), (2, (40, 24, 5)), (3, (5, 9, 6)), (3, (16, 8, 3))]
LENGTH, FACES = (1.1, 0.9, 1.3), 0b100010


def placed(v, offset, dtype):
    import torch

    buf = torch.full((len(v) + offset,), float("nan"), dtype=dtype, device="cuda")
    buf[offset:] = to_gpu(v, dtype)
    return buf[offset:]


def check_modes(g, om, cm, apply):
    """vmult in both precisions at every offset, vmult_add and residual; FP64 1e-12, FP32 2e-6 as in every apply test."""
    import torch

    x, b = uniform_dofs(om, seed=4), uniform_dofs(om, seed=5)
    ref = apply(x)
    free = np.ones(om.ndofs, bool) if cm is None else cm == 0
    for offset in range(4):
        for dtype, tol in ((torch.float64, 1e-12), (torch.float32, 2e-6)):
            y = placed(np.full(om.ndofs, np.nan), offset, dtype)
            g.vmult(y, placed(x, offset, dtype))
            assert rel_err(y.cpu().numpy(), ref) <= tol, (offset, dtype)
    y = placed(b, 1, torch.float64)
    g.vmult_add(y, placed(x, 3, torch.float64), -0.5)
    assert rel_err(y.cpu().numpy(), b - 0.5 * np.where(free, ref, 0.0)) <= 1e-12
    r = placed(np.zeros(om.ndofs), 3, torch.float64)
    g.residual(r, placed(b, 2, torch.float64), placed(x, 1, torch.float64))
    assert rel_err(r.cpu().numpy(), b - np.where(free, ref, 0.0)) <= 1e-12
    assert g.device_errors() == 0


def flags(om, masked):
    return (np.random.default_rng(7).random(om.ndofs) < 0.2).astype(np.uint8) if masked else None


def geometry(degree, m, masked):
    om, _, _ = meshes(degree, m, length=LENGTH)
    return meshes(degree, m, faces=FACES, mask=flags(om, masked), length=LENGTH)


@pytest.mark.parametrize("degree,m", MESHES)
@pytest.mark.parametrize("masked", [False, True])
def test_reinitialisation(degree, m, masked):
    import torch

    from meltpooldg_b200.operators import OlssonOperator

    om, gm, cm = geometry(degree, m, masked)
    dt, eps_n, eps_t, tol = 1e-2, 0.05, 0.01, 1e-3
    normal = [uniform_dofs(om, seed=s) + o for s, o in ((1, 2.0), (2, -1.5), (3, 0.5))]
    g = OlssonOperator(gm, dt=dt, eps_normal=eps_n, eps_tangential=eps_t, normal_tolerance=tol)
    g.set_normal(*[placed(n, s, torch.float64) for n, s in zip(normal, (0, 1, 2))])
    check_modes(g, om, cm, lambda x: oracle_reinit.tangent_apply(om, cm, dt, eps_n, eps_t, normal, tol, x))
    psi = uniform_dofs(om, seed=6)
    for offset in range(2):
        dst = placed(np.full(om.ndofs, np.nan), offset, torch.float64)
        g.create_rhs(dst, placed(psi, offset, torch.float64))
        assert rel_err(dst.cpu().numpy(), oracle_reinit.create_rhs(om, cm, eps_n, eps_t, normal, tol, psi)) <= 1e-12
    assert g.device_errors() == 0


@pytest.mark.parametrize("degree,m", MESHES)
@pytest.mark.parametrize("band", [None, 0.6])
def test_projection(degree, m, band):
    import torch

    from meltpooldg_b200.operators import HeatDiffuseOperator

    om, gm, cm = geometry(degree, m, False)
    g = HeatDiffuseOperator(gm, rho_cp=1.0, dt=1.0, conductivity=0.02)
    X, Y, Z = om.coords()
    psi = np.sin(2.0 * X + 0.3) + 0.7 * Y * Y - 0.5 * Z + 0.2
    level = placed(psi, 1, torch.float64)
    if band:
        g.set_narrow_band(level, band)
        check_modes(g, om, cm, lambda x: oracle_reinit.projection_apply(om, cm, 0.02, x, level_set=psi, narrow_band=band))
    for normalized in (False, True):
        want = oracle_reinit.normal_rhs(om, cm, psi, normalized, narrow_band=band)
        start = [uniform_dofs(om, seed=s) for s in (1, 2, 3)]
        out = [placed(s, o, torch.float64) for s, o in zip(start, (0, 1, 3))]
        g.level_set_normal_rhs(level, *out, normalized=normalized)
        for o, s, w in zip(out, start, want):  # accumulating
            assert rel_err(o.cpu().numpy(), s + w) <= 1e-12
    normal = [uniform_dofs(om, seed=s) + 0.2 for s in (4, 5, 6)]
    dst = placed(np.full(om.ndofs, np.nan), 1, torch.float64)
    g.level_set_curvature_rhs(dst, *[placed(n, 1, torch.float64) for n in normal], 1e-10)
    assert rel_err(dst.cpu().numpy(), oracle_reinit.curvature_rhs(om, cm, normal, 1e-10, level_set=psi, narrow_band=band)) <= 1e-12
    assert g.device_errors() == 0


@pytest.mark.parametrize("degree,m", MESHES)
@pytest.mark.parametrize("masked", [False, True])
def test_solidification(degree, m, masked):
    import torch

    from meltpooldg_b200.operators import HeatDiffuseOperator

    om, gm, cm = geometry(degree, m, masked)
    dt, liquid, solid, liquidus, solidus = 1e-3, (4.1, 0.83, 0.03), (4.4, 0.7, 0.025), 1700.0, 1600.0
    g = HeatDiffuseOperator(gm, rho_cp=1.0, dt=dt, conductivity=1.0)
    g.set_solidification(liquid, solid, liquidus, solidus)
    mat = oracle_solid.SolidLiquid(liquid, solid, liquidus, solidus, False)
    T = 1650.0 + 90.0 * uniform_dofs(om, seed=1)
    old = T - 5.0 * (uniform_dofs(om, seed=2) + 1.0)
    Td, od = placed(T, 1, torch.float64), placed(old, 2, torch.float64)
    g.set_temperature(Td)
    g.set_old_temperature(od)
    check_modes(g, om, cm, lambda x: oracle_solid.tangent_apply(om, cm, mat, dt, T, old, x))
    base = uniform_dofs(om, seed=3)
    dst = placed(base, 3, torch.float64)
    g.create_rhs(dst, Td, od)
    assert rel_err(dst.cpu().numpy(), base + oracle_solid.residual(om, cm, mat, dt, T, old)) <= 1e-12
    d = oracle_solid.diagonal(om, cm, mat, dt, T, old)
    if cm is not None:
        d[cm != 0] = 1.0
    inv = placed(np.full(om.ndofs, np.nan), 1, torch.float64)
    g.compute_inverse_diagonal_from_matrixfree(inv)
    assert rel_err(inv.cpu().numpy(), np.where(np.abs(d) > 1e-10, 1.0 / d, 1.0)) <= 1e-12
    assert g.device_errors() == 0
