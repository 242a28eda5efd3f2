"""Calls on one thread while another captures a stream of the device: they wait
for their own streams only, and the capture goes on."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob(gs):
    a = gs.varcoef_loguniform(15, 16, 17, seed=3)
    return a, gs.Hierarchy.build(a, 1, 0.1, 10, 60), gs.uniform_rhs(a.rows, 1)


@pytest.mark.parametrize("call", ["solve", "update_matrix", "batch"])
def test_beside_a_capture(gs, device, prob, call):
    torch = pytest.importorskip("torch")
    a, H, b = prob
    s = gs.Solver(H, gs.SolverOptions(coarse_tail=0), device=device)
    if call == "update_matrix":
        s.update_matrix(a.val * 2.0)
    want = s.solve(b)[0]
    s.update_matrix(a.val)
    got, errors = [], []

    def run():
        try:
            if call == "batch":
                got.append(gs.Batch([H, H], 1, gs.SolverOptions(), device=device))
            elif call == "update_matrix":
                s.update_matrix(a.val * 2.0)
            got.append(s.solve(b)[0])
        except Exception as e:  # reported below, outside the capture
            errors.append(e)

    t, g = torch.zeros(8, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        t += 1
        th = threading.Thread(target=run)
        th.start()
        th.join()
        t += 1
    g.replay()
    torch.cuda.synchronize()
    assert not errors and bool((t == 2).all())
    assert np.array_equal(got[-1], want)
