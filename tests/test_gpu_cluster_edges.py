"""Edges of the cluster-resident smoothing steps (cluster.cuh), against colour
passes with the same lanes per row: the same bits."""
import numpy as np
import pytest

from test_gpu_cluster import solver_with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_own_values_are_read_before_they_are_replaced(gs, device, tmp_path, precision):
    """Weights that differ from row to row, some exactly 1: the rows of a warp
    part ways around the read of their old values."""
    a = gs.elasticity(9)
    H = gs.Hierarchy.build(a, 3, 0.1, 10, 60)
    out = []
    for cluster in (False, True):
        o = gs.SolverOptions(smoother=1, tol=1e-9, coarse_tail=0, precision=precision, flexible=precision)
        s = solver_with(gs, device, tmp_path, H, o, cluster)
        n = len(s.node_features())
        s.set_node_weights(np.where(np.arange(n) % 3 == 0, 1.0, 0.8 + 0.4 * (np.arange(n) % 7) / 6))
        out.append([s.solve(a.rhs)[0] for _ in range(4)])
    for p in out[0] + out[1]:
        assert np.array_equal(p, out[0][0])


@pytest.fixture
def withheld(gs):
    """While the returned function is on, cluster steps wait for a message that nobody sends."""
    yield gs.lib().gs_debug_withhold_cluster_message
    gs.lib().gs_debug_withhold_cluster_message(0)


@pytest.fixture(scope="module")
def kuhn(gs):
    a = gs.kuhn_laplacian(15)
    return a, gs.Hierarchy.build(a, 1, 0.1, 10, 20), gs.uniform_rhs(a.rows, 5)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("kw", [dict(), dict(pre_steps=2, post_steps=2), dict(half_sweeps=1, coloring=2)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "default")
def test_a_wait_that_gives_up_is_an_error(gs, device, tmp_path, withheld, kuhn, graph, kw):
    """The step returns, the solve reports the failure, and the device goes on."""
    a, H, b = kuhn
    o = gs.SolverOptions(tol=1e-9, coarse_tail=0, use_graph=graph, **kw)
    good = solver_with(gs, device, tmp_path, H, o, True)
    x, _ = good.solve(b)
    withheld(1)
    s = solver_with(gs, device, tmp_path, H, o, True)
    withheld(0)
    for _ in range(2):
        with pytest.raises(gs.SolverError, match="timed out"):
            s.solve(b)
    assert np.array_equal(good.solve(b)[0], x)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("max_iter", [1, 50])
def test_x_is_left_alone_after_a_fault(gs, device, tmp_path, withheld, kuhn, graph, max_iter):
    """The wait gives up in the V-cycle that starts the solve."""
    torch = pytest.importorskip("torch")
    a, H, b = kuhn
    o = gs.SolverOptions(tol=1e-9, coarse_tail=0, use_graph=graph, max_iter=max_iter)
    withheld(1)
    s = solver_with(gs, device, tmp_path, H, o, True)
    bd = torch.from_numpy(np.asarray(b)).cuda()
    x = torch.full_like(bd, 2.0)
    torch.cuda.synchronize()
    with pytest.raises(gs.SolverError, match="timed out"):
        s.solve_device(bd.data_ptr(), x.data_ptr(), 0)
    assert bool((x == 2.0).all())


@pytest.mark.parametrize("precision", [0, 1])
def test_applying_the_preconditioner_reports_a_fault(gs, device, tmp_path, withheld, kuhn, precision):
    torch = pytest.importorskip("torch")
    a, H, b = kuhn
    o = gs.SolverOptions(coarse_tail=0, precision=precision)
    good = solver_with(gs, device, tmp_path, H, o, True)
    withheld(1)
    s = solver_with(gs, device, tmp_path, H, o, True)
    r = torch.from_numpy(np.asarray(b)).cuda()
    z = torch.full_like(r, 2.0)
    torch.cuda.synchronize()
    for _ in range(2):
        with pytest.raises(gs.SolverError, match="timed out"):
            s.apply_preconditioner_device(r.data_ptr(), z.data_ptr(), 0)
        assert bool((z == 2.0).all())
        with pytest.raises(gs.SolverError, match="timed out"):
            s.error_reduction(r.data_ptr(), 0)
    good.apply_preconditioner_device(r.data_ptr(), z.data_ptr(), 0)
    assert bool(torch.isfinite(z).all()) and good.error_reduction(r.data_ptr(), 0) < 1.0


@pytest.mark.parametrize("graph", [0, 1])
def test_the_tuner_drops_a_cluster_whose_wait_gives_up(gs, device, tmp_path, withheld, kuhn, graph):
    """After a fault every launch returns at once: such a step would time as the fastest."""
    a, H, b = kuhn
    o = gs.SolverOptions(tol=1e-9, coarse_tail=0, use_graph=graph)
    path = tmp_path / "decisions"
    gs.set_tune_cache(str(path))
    withheld(1)
    try:
        s = gs.Solver(H, o, device=device)
    finally:
        gs.set_tune_cache(None)
    fields = [int(v) for v in path.read_text().split()[1:]]
    assert not any(fields[6::7])
    x, st = s.solve(b)
    assert st.status == gs.STATUS_CONVERGED and np.linalg.norm(b - a.to_scipy() @ x) <= 2e-9 * np.linalg.norm(b)


def test_the_batch_tuner_drops_a_cluster_whose_wait_gives_up(gs, device, withheld):
    mats = [gs.varcoef_loguniform(x, y, z, seed=3 + i) for i, (x, y, z) in enumerate([(17, 19, 15), (21, 9, 23), (14, 14, 14)])]
    hs = [gs.Hierarchy.build(m, 1, 0.1, 10, 60) for m in mats]
    b = np.concatenate([gs.uniform_rhs(m.rows, i) for i, m in enumerate(mats)])
    withheld(1)
    B = gs.Batch(hs, 1, gs.SolverOptions(tol=1e-9), device=device)
    x, st = B.solve(b)
    assert all(s.status == gs.STATUS_CONVERGED for s in st)
    for m, xi, bi in zip(mats, np.split(x, np.cumsum([m.rows for m in mats])[:-1]),
                         np.split(b, np.cumsum([m.rows for m in mats])[:-1])):
        assert np.linalg.norm(bi - m.to_scipy() @ xi) <= 2e-9 * np.linalg.norm(bi)


def test_the_error_names_the_cluster_step(gs, device, tmp_path, withheld, kuhn):
    a, H, b = kuhn
    withheld(1)
    s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(coarse_tail=0), True)
    with pytest.raises(gs.SolverError, match="cluster Gauss-Seidel step: a wait timed out"):
        s.solve(b)


@pytest.mark.parametrize("precision,exponents", [(0, [-300, -290, -200, 0, 300]), (1, [-37, -34, -31, -20, 0, 37])])
def test_quotients_near_the_ends_of_the_range(gs, device, tmp_path, kuhn, precision, exponents):
    """One V-cycle of right-hand sides whose quotients or their residuals leave
    the normal range, and one with zeros: the bits of the passes' division."""
    torch = pytest.importorskip("torch")
    a, H, b = kuhn
    o = gs.SolverOptions(coarse_tail=0, precision=precision)
    pair = [solver_with(gs, device, tmp_path, H, o, cluster) for cluster in (False, True)]
    for e in exponents + ["zeros"]:
        r = np.where(np.arange(a.rows) % 5 == 0, b, 0.0) if e == "zeros" else b * 10.0 ** e
        rd = torch.from_numpy(r).cuda()
        z = [torch.zeros_like(rd) for _ in pair]
        torch.cuda.synchronize()
        for s, zd in zip(pair, z):
            s.apply_preconditioner_device(rd.data_ptr(), zd.data_ptr(), 0)
        assert np.array_equal(z[0].cpu().numpy(), z[1].cpu().numpy(), equal_nan=True), e
        assert e in (-37, -300) or bool(z[0].any())
