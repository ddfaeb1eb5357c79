"""create_rhs of the heat operator accumulates into dst = T_old or dst = q as into any other vector: every input is
read before dst is added to."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from tests.gpu_util import rel_err, to_gpu
from tests.test_gpu_heat import heat_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,m", [(1, (70, 33, 40)), (2, (40, 17, 30)), (3, (17, 9, 8))])
@pytest.mark.parametrize("into", ["old", "q", "part of q"])
def test_rhs_into_an_input(degree, m, into):
    import torch

    o, g, om, cm = heat_pair(degree, m, faces=0b010100, length=(1.1, 0.9, 1.3))
    T, old, q = (uniform_dofs(om, seed=s) for s in (1, 2, 3))
    shift = 5 if into == "part of q" else 0
    pool = torch.empty(om.ndofs + shift, dtype=torch.float64, device="cuda")
    dst, qd, od = pool[:om.ndofs], to_gpu(q), to_gpu(old)
    if into == "old":
        dst.copy_(od)
        od = dst
    else:
        pool[shift:] = qd
        qd = pool[shift:]
        dst[:shift] = 0.0
    ref = dst.cpu().numpy().copy()
    o.create_rhs(ref, T, od.cpu().numpy().copy(), qd.cpu().numpy().copy())
    g.create_rhs(dst, to_gpu(T), od, qd)
    # sums of two products of 27 (64) terms with coefficients up to rho c_p / dt, as without aliasing
    assert rel_err(dst.cpu().numpy(), ref) <= 1e-12
    assert np.isfinite(ref).all() and g.device_errors() == 0
