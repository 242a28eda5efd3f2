"""Batched passes over long and short lists of items (batch.cuh: kHead): the
same systems solved together, where the fine level's lists are long, and one by
one, where they are short; and one system whose slice lists are long."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 4])
@pytest.mark.parametrize("kw", [dict(), dict(omega=0.9), dict(use_graph=1)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "default")
def test_long_row_lists_match_short_ones(gs, device, nrhs, kw):
    """32 lanes a row: 8 rows an item, so 8 x 1184 items are 75,776 rows of a
    colour; 54 x 53 x 55 cells have more in either colour, the others less."""
    sides = [(54, 53, 55), (33, 47, 29), (51, 49, 50)]
    mats = [gs.varcoef_loguniform(*s, seed=3 + i) for i, s in enumerate(sides)]
    hs = [gs.Hierarchy.build(m, 1, 0.1, 10, 1000) for m in mats]
    b = [np.concatenate([gs.uniform_rhs(m.rows, 10 * i + j) for j in range(nrhs)]) for i, m in enumerate(mats)]
    o = gs.SolverOptions(tol=1e-12, lanes=32, **kw)
    x, st = gs.Batch(hs, nrhs, o, device=device).solve(np.concatenate(b))
    assert all(s.status == gs.STATUS_CONVERGED for s in st)
    parts = np.split(x, np.cumsum([v.size for v in b])[:-1])
    for i in range(len(mats)):
        xi, si = gs.Batch([hs[i]], nrhs, o, device=device).solve(b[i])
        # FP64; the products' partial sums are cut elsewhere, so the stop may fall one iteration apart at 1e-12
        assert all(abs(p.iterations - q.iterations) <= 1 for p, q in zip(si, st[nrhs * i:nrhs * (i + 1)]))
        assert np.linalg.norm(parts[i] - xi) <= 1e-9 * np.linalg.norm(xi)


@pytest.mark.parametrize("precision", [0, 1])
def test_long_slice_lists(gs, device, precision):
    """One lane a row: 4 x 1184 items of 8 slices are 1,212,416 rows of a colour."""
    a = gs.varcoef_loguniform(140, 138, 139, seed=2)
    H = gs.Hierarchy.build_ex(a, 1, 0.1, 10, 1000, aggregation=1, device=device)
    b = gs.uniform_rhs(a.rows, 5)
    o = gs.SolverOptions(tol=1e-9, lanes=1, precision=precision, flexible=precision, max_iter=400)
    x, st = gs.Batch([H], 1, o, device=device).solve(b)
    assert st[0].status == gs.STATUS_CONVERGED
    # the recurrence's residual has left the true one by far less than the tolerance
    assert np.linalg.norm(b - a.to_scipy() @ x) <= 2e-9 * np.linalg.norm(b)
    _, ref = gs.Solver(H, gs.SolverOptions(tol=1e-9, coarse_tail=0, precision=precision, flexible=precision, max_iter=400),
                       device=device).solve(b)
    assert abs(st[0].iterations - ref.iterations) <= 1
