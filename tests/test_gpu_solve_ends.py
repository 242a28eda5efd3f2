"""How a solve starts and ends, with iterations issued directly and replayed:
stops after a given number of iterations, a zero right-hand side, a start that
has converged already, and values that are not finite, through the host and
the device entry points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob(gs):
    a = gs.varcoef_loguniform(9, 10, 11, seed=3)
    return a, gs.Hierarchy.build(a, 1, 0.1, 10, 40), gs.uniform_rhs(a.rows, 4)


def solver(gs, device, prob, graph, **kw):
    return gs.Solver(prob[1], gs.SolverOptions(coarse_tail=0, use_graph=graph, **kw), device=device)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("max_iter", [1, 2, 3, 4])
def test_max_iter(gs, orc, device, prob, graph, max_iter):
    a, H, b = prob
    n = H.levels
    A, P, R = [H.A(k) for k in range(n)], [H.P(k) for k in range(n - 1)], [H.R(k) for k in range(n - 1)]
    x, st = solver(gs, device, prob, graph, tol=1e-14, max_iter=max_iter).solve(b)
    xo, it, status, _ = orc.amg_pcg(A, P, R, b, tol=1e-14, max_iter=max_iter)
    assert st.status == gs.STATUS_MAX_ITER and st.iterations == max_iter == it
    # FP64, the same operations up to the order of a row's sum: a few hundred roundings an iteration
    assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)


@pytest.mark.parametrize("graph", [0, 1])
def test_device_solves_that_end_at_the_start(gs, device, prob, graph):
    torch = pytest.importorskip("torch")
    a, H, b = prob
    first, _ = solver(gs, device, prob, graph, tol=1e-11).solve(b)  # well below the stop of the solver under test
    s = solver(gs, device, prob, graph, tol=1e-8)
    own, _ = s.solve(b)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        bd = torch.from_numpy(np.asarray(b)).cuda()
        x = torch.full_like(bd, 3.0)
        zero = torch.zeros_like(bd)
        st = s.solve_device(zero.data_ptr(), x.data_ptr(), stream.cuda_stream)
        assert st.status == gs.STATUS_ZERO_RHS and not x.any()
        x.copy_(torch.from_numpy(first))
        st = s.solve_device(bd.data_ptr(), x.data_ptr(), stream.cuda_stream)
        assert st.status == gs.STATUS_INITIAL_CONVERGED and st.iterations == 0
        assert np.array_equal(x.cpu().numpy(), first)
        bad = bd.clone()
        bad[7] = float("inf")
        x.fill_(2.0)
        with pytest.raises(gs.NotFiniteError):
            s.solve_device(bad.data_ptr(), x.data_ptr(), stream.cuda_stream)
        assert bool((x == 2.0).all())
        x.zero_()
        st = s.solve_device(bd.data_ptr(), x.data_ptr(), stream.cuda_stream)
        assert st.status == gs.STATUS_CONVERGED and np.array_equal(x.cpu().numpy(), own)
