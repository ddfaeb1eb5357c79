"""Advection apply and heat apply with a convection velocity in columns of 16 x 8 cells (meshes that would leave a fifth
of the wider columns' threads without a cell): one and several columns, partial in x and y, per-DoF flags, every element
offset and each output mode, against the oracles."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from oracle import advection_field
from oracle.oracle import Operator as OOp
from tests.gpu_util import meshes, to_gpu
from tests.test_gpu_advection_march import DT, EPS, THETA, VEL
from tests.test_gpu_point_march import check_modes

pytestmark = pytest.mark.gpu

MESHES = [(1, (8, 17, 30)), (1, (40, 24, 5)), (2, (5, 9, 6)), (2, (16, 8, 3)), (2, (40, 24, 5)), (3, (5, 9, 6)), (3, (17, 16, 3))]


@pytest.mark.parametrize("degree,m", MESHES)
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("field", [False, True])
def test_narrow_columns(degree, m, masked, field):
    from meltpooldg_b200.operators import AdvectionDiffusionOperator

    n = np.prod([degree * c + 1 for c in m])
    mask = (np.random.default_rng(7).random(n) < 0.2).astype(np.uint8) if masked else None
    om, gm, cm = meshes(degree, m, faces=0b100010, mask=mask, length=(1.0, 0.9, 1.2))
    g = AdvectionDiffusionOperator(gm, dt=DT, theta=THETA, diffusivity=EPS, velocity=VEL)
    if field:
        v = [uniform_dofs(om, seed=s) for s in (1, 2, 3)]
        vd = [to_gpu(c) for c in v]
        g.set_velocity_field(*vd)
        apply = lambda x: advection_field.tangent_apply(om, cm, v, DT, THETA, EPS, x)  # noqa: E731
    else:
        apply = OOp(om, "advdiff", cmask=cm, dt=DT, theta=THETA, eps=EPS, vel=VEL).vmult
    check_modes(g, om, cm, lambda x: np.where(cm == 0, apply(x), 0.0))
