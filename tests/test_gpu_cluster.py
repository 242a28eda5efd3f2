"""Smoothing steps of a small level in one thread-block cluster (cluster.cuh)
against one launch per colour pass with the same lanes per row: the same bits.
The autotuner picks the launch mode by timing, so the test writes the decision
file itself: CSR-vector layouts with the lanes the cluster uses, cluster
steps off or on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lanes_of(a, block=1):
    """Lanes per row of a level in the cluster (about five entries, or two 3x3 blocks, a lane)."""
    length, g = a.nnz / a.rows / block - 1.0, 4
    while g < 32 and g * (2.0 if block == 3 else 5.0) < length:
        g *= 2
    return g


def solver_with(gs, device, tmp_path, H, opts, cluster, mask=None):
    """A solver whose decision file says `cluster` for every level (or mask[k])."""
    path = tmp_path / "tune"
    gs.set_tune_cache(str(path))
    try:
        if path.exists():
            path.unlink()
        levels = len(gs.Solver(H, opts, device=device).level_info())
        key = [ln.split()[0] for ln in path.read_text().splitlines() if ln.startswith("v5:")][0]
        fields = []
        for k in range(levels):
            on = cluster and (mask is None or mask[k])
            fields += [0, lanes_of(H.A(k), 3 if opts.smoother == 1 else 1), 8, 4, 0, 0, int(on)]
        path.write_text(key + " " + " ".join(map(str, fields)) + " 1\n")
        return gs.Solver(H, opts, device=device)
    finally:
        gs.set_tune_cache(None)


def problems(gs):
    grf = gs.varcoef_grf(20, 8.0, 2.3, 4)
    kuhn = gs.kuhn_laplacian(15)
    return {"grf20": (grf, gs.Hierarchy.build(grf, 1, 0.1, 10, 60)),
            "kuhn15": (kuhn, gs.Hierarchy.build(kuhn, 1, 0.1, 10, 20))}


@pytest.fixture(scope="module")
def probs(gs):
    return problems(gs)


@pytest.mark.parametrize("name", ["grf20", "kuhn15"])
@pytest.mark.parametrize("kw", [
    dict(),
    dict(use_graph=1, flexible=1, precision=1),
    dict(omega=0.8, pre_steps=2, post_steps=1, vcycles=2),
    dict(half_sweeps=1, coloring=1),
    dict(half_sweeps=1, coloring=2, precision=1, flexible=1, pre_steps=2, post_steps=2),
    dict(coloring=2),
    dict(overlap_launch=0),
    dict(coarse_solver=0, coarse_steps=3),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "default")
def test_cluster_steps_are_bit_identical(gs, device, tmp_path, probs, name, kw):
    a, H = probs[name]
    b = gs.uniform_rhs(a.rows, 3)
    out = []
    for cluster in (False, True):
        s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(tol=1e-9, coarse_tail=0, **kw), cluster)
        launch = [lv["launch"] for lv in s.level_info()]
        assert any(launch) == cluster
        x, st = s.solve(b)
        again, _ = s.solve(b)
        assert st.status == gs.STATUS_CONVERGED and np.array_equal(x, again)
        out.append((x, st.iterations))
    assert out[0][1] == out[1][1] and np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("side,min_dofs", [(4, 20), (9, 60)])
@pytest.mark.parametrize("kw", [
    dict(),
    dict(use_graph=1, flexible=1, precision=1),
    dict(omega=0.9, pre_steps=2, post_steps=1),
    dict(half_sweeps=1, coloring=2, precision=1, flexible=1),
    dict(half_sweeps=1, coloring=2, pre_steps=2, post_steps=2),
], ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "default")
def test_block_cluster_steps_are_bit_identical(gs, device, tmp_path, kw, side, min_dofs):
    """3x3 block levels; also with a weight per node and with new values."""
    a = gs.elasticity(side)
    H = gs.Hierarchy.build(a, 3, 0.1, 10, min_dofs)
    out = []
    for cluster in (False, True):
        s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(smoother=1, tol=1e-9, coarse_tail=0, **kw), cluster)
        before = s.launch_count()
        runs = [s.solve(a.rhs)[0]]
        launches = s.launch_count() - before
        if cluster:
            assert launches < passes  # a step is one launch, not one per colour pass
        passes = launches
        n = len(s.node_features())
        s.set_node_weights(np.linspace(0.9, 1.1, n))
        runs.append(s.solve(a.rhs)[0])
        s.set_node_weights(None)
        s.update_matrix(a.val * 3.0)
        runs.append(s.solve(a.rhs)[0])
        out.append(runs)
    for p, q in zip(*out):
        assert np.array_equal(p, q)


def test_cluster_steps_with_weights_and_refresh(gs, device, tmp_path, probs):
    """Colour weights (read per pass) and new matrix values of the same pattern."""
    a, H = probs["kuhn15"]
    b = gs.uniform_rhs(a.rows, 5)
    out = []
    for cluster in (False, True):
        s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(tol=1e-9, coarse_tail=0), cluster)
        runs = [s.solve(b)[0]]
        s.set_colour_weights([np.linspace(0.9, 1.1, lv["colors"]) for lv in s.level_info()])
        runs.append(s.solve(b)[0])
        s.set_colour_weights(None)
        s.update_matrix(H.A(0).val * 2.5)
        runs.append(s.solve(b)[0])
        out.append(runs)
    for p, q in zip(*out):
        assert np.array_equal(p, q)
    assert np.linalg.norm(out[1][2] * 2.5 - out[1][0]) <= 1e-7 * np.linalg.norm(out[1][0])


def test_unsuitable_levels_keep_their_passes(gs, device, tmp_path):
    """A level whose 16 CTAs would need more slots than shared memory holds
    (random couplings over 60,000 rows: every CTA reads almost every row) is
    refused when the layout is built, whatever the decision file says."""
    n = 60000
    r = np.random.default_rng(2)
    import scipy.sparse as sp
    i, j = r.integers(0, n, 400000), r.integers(0, n, 400000)
    w = sp.coo_matrix((np.ones(len(i)), (i, j)), shape=(n, n))
    w = ((w + w.T) > 0).astype(np.float64).tocsr()
    w.setdiag(0)
    w.eliminate_zeros()
    m = gs.Csr.from_scipy(sp.diags(np.asarray(w.sum(1)).ravel() + 1.0) - w)
    p = sp.csr_matrix((np.ones(n), (np.arange(n), np.arange(n) % 50)), shape=(n, 50))
    A = m.to_scipy()
    H = gs.Hierarchy.from_levels([m, gs.Csr.from_scipy(p.T @ A @ p)], [gs.Csr.from_scipy(p)], [gs.Csr.from_scipy(p.T)])
    s = solver_with(gs, device, tmp_path, H, gs.SolverOptions(tol=1e-8, coarse_tail=0), True)
    assert s.level_info()[0]["launch"] == 0
    b = gs.uniform_rhs(n, 1)
    x, st = s.solve(b)
    assert st.status == gs.STATUS_CONVERGED
    assert np.linalg.norm(b - A @ x) <= 2e-8 * np.linalg.norm(b)
