"""Krylov solvers where their host and launch plans change: small lattices of the one-launch CG (one low piece per
CTA), GMRES restarts of every length class, without a preconditioner, and stopped by the iteration limit."""
import numpy as np
import pytest

from meltpooldg_b200.inputs import uniform_dofs
from tests.gpu_util import to_gpu
from tests.test_gpu_advdiff import adv_pair
from tests.test_gpu_heat import heat_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [(5, 3, 1), (16, 16, 16), (33, 9, 21), (64, 40, 37), (96, 17, 66)])
def test_fused_cg_on_small_lattices(m):
    import torch

    from meltpooldg_b200 import _lib as L
    from meltpooldg_b200.operators import LinearSolver, LinearSolverData

    o, g, om, cm = heat_pair(2, m)
    b = uniform_dofs(om, seed=3, cmask=cm)
    data, its = LinearSolverData("CG", "Diagonal", rel_tolerance=1e-11), []
    for variant in (1, 0):
        assert L.lib().mpdg_op_set_cg_variant(g._h, variant) == L.MPDG_OK
        x = torch.zeros(om.ndofs, dtype=torch.float64, device="cuda")
        st = LinearSolver.solve(g, x, to_gpu(b), data)
        its.append(st.iterations)
        # the recursive residual follows the true one to a few digits above rounding
        assert np.linalg.norm(b - o.vmult(x.cpu().numpy())) <= 2e-11 * np.linalg.norm(b)
    assert abs(its[0] - its[1]) <= 1
    x32 = torch.zeros(om.ndofs, dtype=torch.float64, device="cuda")
    LinearSolver.solve_mixed(g, x32, to_gpu(b), outer_rel_tol=1e-11, inner_rel_tol=1e-5)
    assert np.linalg.norm(b - o.vmult(x32.cpu().numpy())) <= 2e-11 * np.linalg.norm(b)
    assert g.device_errors() == 0


@pytest.mark.parametrize("restart", [1, 2, 7, 31])
@pytest.mark.parametrize("precond", ["Identity", "Diagonal"])
def test_gmres_restarts(restart, precond):
    import torch

    from meltpooldg_b200.operators import LinearSolver, LinearSolverData, NoConvergence

    o, g, om, cm = adv_pair(2, (9, 8, 5), faces=0b000011)
    b = uniform_dofs(om, seed=5, cmask=cm)
    x = torch.zeros(om.ndofs, dtype=torch.float64, device="cuda")
    st = LinearSolver.solve(g, x, to_gpu(b), LinearSolverData("GMRES", precond, rel_tolerance=1e-9, restart=restart), history=True)
    assert len(st.history) == st.iterations + 1 and np.all(np.isfinite(st.history))
    assert np.linalg.norm(b - o.vmult(x.cpu().numpy())) <= 2e-9 * np.linalg.norm(b)
    x.zero_()
    with pytest.raises(NoConvergence):
        LinearSolver.solve(g, x, to_gpu(b), LinearSolverData("GMRES", precond, rel_tolerance=1e-9, restart=restart, max_iterations=3))
    # the three iterations' update reached x
    assert 0.0 < np.linalg.norm(b - o.vmult(x.cpu().numpy())) < np.linalg.norm(b)
