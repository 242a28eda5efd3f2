"""Kernels that load operands before they wait on the launch ahead of them: the
same bits whether launches overlap or not, where only few launches lie between
a vector's writer and its reader."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 70001])
@pytest.mark.parametrize("flexible", [0, 1])
def test_one_level_of_one_colour(gs, device, n, flexible):
    """A diagonal matrix: one level, one colour, so the whole preconditioner is
    one pass. FP32 passes and a tight tolerance keep the solve going past its
    first iteration."""
    r = np.random.default_rng(n)
    d = r.uniform(0.5, 3.0, n) if n > 1 else np.array([3.0])
    H = gs.Hierarchy.from_levels([gs.Csr.from_scipy(sp.diags(d).tocsr())], [], [])
    b = gs.uniform_rhs(n, 5)
    out = []
    for graph in (0, 1):
        for overlap in (0, 1, 2):
            o = gs.SolverOptions(tol=1e-13, precision=1, flexible=flexible, coarse_solver=0, coarse_tail=0,
                                 use_graph=graph, overlap_launch=overlap)
            s = gs.Solver(H, o, device=device)
            for _ in range(3):
                x, st = s.solve(b)
                out.append((x, st.iterations, st.status))
            # FP32 relaxation: 24 bits an iteration at least
            assert st.status == gs.STATUS_CONVERGED and np.linalg.norm(d * x - b) <= 2e-13 * np.linalg.norm(b)
    for x, it, status in out[1:]:
        assert it == out[0][1] and status == out[0][2] and np.array_equal(x, out[0][0])


@pytest.mark.parametrize("graph", [0, 1])
def test_a_zero_right_hand_side_stops_at_the_start(gs, device, graph):
    """The iteration queued behind the start does not run: the statistics are
    those of the start, x0 = 1 and b below the bound of a zero right-hand side."""
    a = gs.varcoef_loguniform(9, 10, 11, seed=3)
    s = gs.Solver(gs.Hierarchy.build(a, 1, 0.1, 10, 40), gs.SolverOptions(tol=1e-8, coarse_tail=0, use_graph=graph),
                  device=device)
    b, x0 = np.full(a.rows, 1e-18), np.ones(a.rows)
    x, st = s.solve(b, x0)
    assert st.status == gs.STATUS_ZERO_RHS and st.iterations == 0 and st.spmv == 0 and not x.any()
    # sums of 990 squares in FP64
    assert st.rhs_norm2 == pytest.approx(float(b @ b), rel=1e-12)
    r = b - a.to_scipy() @ x0
    assert st.ratio == pytest.approx(float(r @ r) / float(b @ b), rel=1e-10)


@pytest.mark.parametrize("tail", [0, 2])
def test_weights_count_from_the_next_solve(gs, device, tail):
    """Weights of two kinds in turn, each solved with at once."""
    a = gs.varcoef_loguniform(17, 16, 15, seed=3)
    s = gs.Solver(gs.Hierarchy.build(a, 1, 0.1, 10, 60), gs.SolverOptions(tol=1e-9, coarse_tail=tail), device=device)
    b = gs.uniform_rhs(a.rows, 2)
    n = [lv["colors"] for lv in s.level_info()]
    kinds = [[np.linspace(0.9, 1.1, c) for c in n], [np.full(c, 0.85) for c in n], None]
    want = [None] * 3
    for i in range(24):
        s.set_colour_weights(kinds[i % 3])
        x, st = s.solve(b)
        assert st.status == gs.STATUS_CONVERGED
        want[i % 3] = x if want[i % 3] is None else want[i % 3]
        assert np.array_equal(x, want[i % 3])
    assert not np.array_equal(want[0], want[1])
