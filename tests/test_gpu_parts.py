"""The parts of a V-cycle level that the smoother makes unnecessary (the colour
solved last has no residual, the colour swept first needs no correction, a
sweep from zero uses half of the matrix) against the oracle, over layouts,
colour counts and the options that switch the parts off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def levels(H):
    n = H.levels
    return [H.A(k) for k in range(n)], [H.P(k) for k in range(n - 1)], [H.R(k) for k in range(n - 1)]


def rel(x, y):
    return float(np.linalg.norm(x - y) / np.linalg.norm(y))


@pytest.fixture(scope="module")
def probs(gs):
    p = gs.varcoef_loguniform(9, 14, 11, seed=5)       # two colours, ragged last slices
    k = gs.kuhn_laplacian(11)                          # eight colours
    e = gs.elasticity(7)                               # 3x3 blocks
    return {"poisson": (p, gs.Hierarchy.build(p, 1, 0.1, 10, 40), gs.uniform_rhs(p.rows, 2), 0),
            "kuhn": (k, gs.Hierarchy.build(k, 1, 0.1, 10, 40), gs.uniform_rhs(k.rows, 2), 0),
            "elast": (e, gs.Hierarchy.build(e, 3, 0.1, 10, 60), e.rhs, 1)}


@pytest.mark.parametrize("name", ["poisson", "kuhn", "elast"])
@pytest.mark.parametrize("half,pre,post,vcycles", [(0, 1, 1, 1), (1, 1, 1, 1), (1, 2, 1, 1), (0, 2, 2, 1), (1, 1, 1, 2)])
@pytest.mark.parametrize("layout", [dict(lanes=1), dict(lanes=8), dict(lanes=32), dict(sliced_lanes=4), dict()],
                         ids=["l1", "l8", "l32", "s4", "tuned"])
def test_solve_matches_oracle(gs, orc, device, probs, name, half, pre, post, vcycles, layout):
    a, H, b, smoother = probs[name]
    A, P, R = levels(H)
    kw = dict(pre=pre, post=post, vcycles=vcycles, half_sweeps=half)
    s = gs.Solver(H, gs.SolverOptions(smoother=smoother, tol=1e-9, coarse_tail=0, pre_steps=pre, post_steps=post,
                                      vcycles=vcycles, half_sweeps=half, **layout), device=device)
    x, st = s.solve(b)
    xo, it, status, _ = orc.amg_pcg(A, P, R, b, smoother=smoother, tol=1e-9, **kw)
    assert status == 1 and abs(st.iterations - it) <= 1 and rel(x, xo) <= 1e-10
    # weights of exactly 1 keep the parts, others switch them off and back on
    if smoother == 0 and half == 0:
        n = [lv["colors"] for lv in s.level_info()]
        s.set_colour_weights([np.linspace(0.9, 1.1, c) for c in n])
        xw, _ = s.solve(b)
        xwo, _, _, _ = orc.amg_pcg(A, P, R, b, smoother=0, tol=1e-9, weights=[np.linspace(0.9, 1.1, c) for c in n], **kw)
        assert rel(xw, xwo) <= 1e-10
        s.set_colour_weights(None)
        assert np.array_equal(s.solve(b)[0], x)
