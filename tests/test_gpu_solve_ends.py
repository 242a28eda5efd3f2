"""How a solve starts and ends, with iterations issued directly and replayed:
stops after a given number of iterations, a zero right-hand side, a start that
has converged already, and values that are not finite, through the host and
the device entry points."""
import ctypes

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


@pytest.mark.parametrize("overlap", [0, 1, 2])
@pytest.mark.parametrize("graph", [0, 1])
def test_batch_ends(gs, orc, device, graph, overlap):
    mats = [gs.varcoef_loguniform(x, y, z, seed=7 + i) for i, (x, y, z) in enumerate([(9, 5, 7), (13, 13, 13), (5, 7, 11)])]
    hs = [gs.Hierarchy.build(m, 1, 0.1, 10, 60) for m in mats]
    n = [m.rows for m in mats]
    at = np.concatenate([[0], np.cumsum(n)])

    def batch(**kw):
        return gs.Batch(hs, 1, gs.SolverOptions(use_graph=graph, overlap_launch=overlap, **kw), device=device)

    b = np.concatenate([gs.uniform_rhs(m, i) for i, m in enumerate(n)])
    for max_iter in (1, 2, 5):
        x, st = batch(tol=1e-14, max_iter=max_iter).solve(b)
        for i, H in enumerate(hs):
            L = H.levels
            xo, _, _, _ = orc.amg_pcg([H.A(k) for k in range(L)], [H.P(k) for k in range(L - 1)],
                                      [H.R(k) for k in range(L - 1)], b[at[i]:at[i + 1]], tol=1e-14, max_iter=max_iter)
            assert st[i].status == gs.STATUS_MAX_ITER and st[i].iterations == max_iter
            # FP64, the same operations up to the order of a row's sum
            assert np.linalg.norm(x[at[i]:at[i + 1]] - xo) <= 1e-11 * np.linalg.norm(xo)
    B = batch(tol=1e-8, max_iter=200)
    own, st = B.solve(b)
    assert all(s.status == gs.STATUS_CONVERGED for s in st)
    # every system done at the start, then one of three, then none
    x, st = B.solve(np.zeros_like(b), np.ones_like(b))
    assert all(s.status == gs.STATUS_ZERO_RHS for s in st) and not x.any()
    part = b.copy()
    part[at[1]:at[2]] = 0.0
    x, st = B.solve(part, np.zeros_like(b))
    assert [s.status for s in st] == [gs.STATUS_CONVERGED, gs.STATUS_ZERO_RHS, gs.STATUS_CONVERGED]
    assert not x[at[1]:at[2]].any() and np.array_equal(x[:at[1]], own[:at[1]]) and np.array_equal(x[at[2]:], own[at[2]:])
    x, st = B.solve(b)
    assert np.array_equal(x, own)
    x0 = np.linspace(-1.0, 1.0, b.size)
    assert gs.lib().gs_batch_set_tolerance(B._b, ctypes.c_double(1e-8), 0) == 0
    x, st = B.solve(b, x0)
    assert np.array_equal(x, x0) and all(s.iterations == 0 for s in st)
