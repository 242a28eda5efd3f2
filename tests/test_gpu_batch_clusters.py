"""Batched smoothing steps in thread-block clusters, forced, against the colour
passes with the same lanes per row: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def forced(gs):
    """While the returned function is on, batches take clusters of their forced lanes."""
    yield gs.lib().gs_debug_force_batch_clusters
    gs.lib().gs_debug_force_batch_clusters(0)


@pytest.fixture(scope="module")
def systems(gs):
    few = [(17, 19, 15), (21, 9, 23), (14, 14, 14)]
    many = few + [(9, 10, 11), (15, 8, 12), (13, 13, 13), (7, 21, 9), (16, 11, 10), (12, 12, 18), (19, 8, 8), (10, 17, 13)]
    out = {}
    for name, sides in (("few", few), ("many", many)):
        mats = [gs.varcoef_loguniform(*s, seed=3 + i) for i, s in enumerate(sides)]
        out[name] = mats, [gs.Hierarchy.build(m, 1, 0.1, 10, 60) for m in mats]
    return out


def pair(gs, device, forced, hs, nrhs, **kw):
    out = []
    for on in (0, 1):
        forced(on)
        out.append(gs.Batch(hs, nrhs, gs.SolverOptions(tol=1e-9, **kw), device=device))
    forced(0)
    return out


@pytest.mark.parametrize("name,ctas", [("few", 16), ("many", 8)])
@pytest.mark.parametrize("nrhs,precision,lanes", [(1, 0, 8), (2, 0, 4), (3, 0, 16), (4, 0, 8),
                                                  (1, 1, 16), (2, 1, 8), (3, 1, 4), (4, 1, 32)])
def test_clusters_equal_the_passes(gs, device, systems, forced, name, ctas, nrhs, precision, lanes):
    """Clusters of 16 CTAs (up to nine systems) and of 8; also with one system
    that has nothing to do."""
    mats, hs = systems[name]
    passes, clusters = pair(gs, device, forced, hs, nrhs, precision=precision, flexible=precision, lanes=lanes)
    info = clusters.level_info()
    smoothed = [lv["cluster"] for lv in info[1:-1]]
    # a coarser level has fewer systems and may have the wider clusters
    assert smoothed[0] == ctas and all(c in (8, 16) for c in smoothed) and info[0]["cluster"] == 0
    assert not any(lv["cluster"] for lv in passes.level_info())
    b = np.concatenate([gs.uniform_rhs(m.rows, 10 * i + j) for i, m in enumerate(mats) for j in range(nrhs)])
    idle = b.copy()
    idle[mats[0].rows * nrhs:(mats[0].rows + mats[1].rows) * nrhs] = 0.0
    for rhs in (b, idle):
        x, st = passes.solve(rhs)
        y, su = clusters.solve(rhs)
        assert all(s.status in (gs.STATUS_CONVERGED, gs.STATUS_ZERO_RHS) for s in st)
        assert [s.iterations for s in st] == [s.iterations for s in su] and np.array_equal(x, y)


@pytest.mark.parametrize("kw", [dict(omega=0.9), dict(pre_steps=2, post_steps=2), dict(coloring=1), dict(use_graph=1),
                                dict(overlap_launch=0), dict(vcycles=2)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()))
def test_clusters_equal_the_passes_with_options(gs, device, systems, forced, kw):
    mats, hs = systems["few"]
    passes, clusters = pair(gs, device, forced, hs, 2, lanes=8, **kw)
    assert clusters.level_info()[1]["cluster"] == 16
    b = np.concatenate([gs.uniform_rhs(m.rows, 10 * i + j) for i, m in enumerate(mats) for j in range(2)])
    x, st = passes.solve(b)
    y, su = clusters.solve(b)
    assert all(s.status == gs.STATUS_CONVERGED for s in st)
    assert [s.iterations for s in st] == [s.iterations for s in su] and np.array_equal(x, y)


def test_a_fault_in_a_batch_is_reported(gs, device, systems, forced):
    """A wait that gives up ends the batch with an error; x is left alone, and other batches go on."""
    mats, hs = systems["few"]
    good, _ = pair(gs, device, forced, hs, 1, lanes=8)
    forced(1)
    gs.lib().gs_debug_withhold_cluster_message(1)
    try:
        bad = gs.Batch(hs, 1, gs.SolverOptions(tol=1e-9, lanes=8), device=device)
    finally:
        gs.lib().gs_debug_withhold_cluster_message(0)
    assert bad.level_info()[1]["cluster"] == 16
    torch = pytest.importorskip("torch")
    b = np.concatenate([gs.uniform_rhs(m.rows, i) for i, m in enumerate(mats)])
    bd, x = torch.from_numpy(b).cuda(), torch.full((b.size,), 2.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        with pytest.raises(gs.SolverError, match="timed out"):
            bad.solve_device(bd.data_ptr(), x.data_ptr(), 0)
        assert bool((x == 2.0).all())
    want, _ = good.solve(b)
    assert np.array_equal(good.solve(b)[0], want)


def test_level_info_names_the_clusters(gs, device, tmp_path):
    """Scalar and 3x3 levels report the CTAs of their cluster."""
    from test_gpu_cluster import solver_with
    for a, block in ((gs.kuhn_laplacian(12), 1), (gs.elasticity(7), 3)):
        H = gs.Hierarchy.build(a, block, 0.1, 10, 60)
        for on in (False, True):
            o = gs.SolverOptions(smoother=1 if block == 3 else 0, coarse_tail=0)
            info = solver_with(gs, device, tmp_path, H, o, on).level_info()
            assert [lv["cluster"] in (8, 16) for lv in info[:-1]] == [on] * (len(info) - 1)
