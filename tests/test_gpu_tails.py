"""Two solvers whose coarse tails differ in size stay usable side by side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_two_tails(gs, device, graph):
    big, small = gs.varcoef_loguniform(24, 24, 24, seed=1), gs.varcoef_loguniform(10, 9, 8, seed=2)

    def solver(a):
        o = gs.SolverOptions(tol=1e-8, coarse_tail=2, use_graph=graph)
        return gs.Solver(gs.Hierarchy.build(a, 1, 0.1, 10, 40), o, device=device)

    b = [gs.uniform_rhs(a.rows, 3) for a in (big, small)]
    alone = [solver(a).solve(v)[0] for a, v in zip((big, small), b)]
    pair = [solver(big), solver(small)]  # the second, smaller tail is set up last
    for _ in range(2):
        for s, v, x in zip(pair, b, alone):
            got, st = s.solve(v)
            assert st.status == gs.STATUS_CONVERGED
            # tails are timed: another cluster size adds a row's terms in another order
            assert np.linalg.norm(got - x) <= 1e-6 * np.linalg.norm(x)
