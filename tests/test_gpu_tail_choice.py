"""The coarse tail and the cluster steps of the levels it takes."""
import numpy as np
import pytest

from test_gpu_cluster import solver_with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_levels_of_the_tail_hold_no_cluster_layout(gs, device, tmp_path, graph):
    """A forced tail on a decision file that asks for cluster steps: its levels
    drop theirs, and report, solve and refresh as the tail does."""
    a = gs.varcoef_loguniform(17, 16, 15, seed=3)
    H = gs.Hierarchy.build(a, 1, 0.1, 10, 60)
    b = gs.uniform_rhs(a.rows, 2)
    s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(tol=1e-9, coarse_tail=2, use_graph=graph), True)
    info = s.level_info()
    assert any(lv["in_tail"] for lv in info) and info[0]["launch"] == 1 and not info[0]["in_tail"]
    assert all(lv["launch"] == 0 for lv in info if lv["in_tail"])
    x, st = s.solve(b)
    assert st.status == gs.STATUS_CONVERGED and np.linalg.norm(b - a.to_scipy() @ x) <= 2e-9 * np.linalg.norm(b)
    s.update_matrix(a.val * 2.0)
    y, st = s.solve(b)
    assert st.status == gs.STATUS_CONVERGED and np.linalg.norm(b - 2.0 * (a.to_scipy() @ y)) <= 2e-9 * np.linalg.norm(b)
