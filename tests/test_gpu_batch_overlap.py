"""Batched solves with programmatic dependent launch (matrix operands loaded
before the wait on the previous pass) against plain stream order: the same
bits, eager and graph-replayed, for every layout of the colour passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def systems(gs):
    # uneven: one slice and a bit, odd sides, two and three levels
    mats = [gs.varcoef_loguniform(x, y, z, seed=7 + i)
            for i, (x, y, z) in enumerate([(9, 5, 7), (13, 13, 13), (17, 11, 6), (5, 7, 33)])]
    return mats, [gs.Hierarchy.build(m, 1, 0.1, 10, 60) for m in mats]


@pytest.mark.parametrize("nrhs,precision", [(1, 0), (4, 1), (3, 0)])
@pytest.mark.parametrize("lanes", [1, 2, 8, 32])
def test_overlapped_batch_is_bit_identical(gs, device, systems, nrhs, precision, lanes):
    mats, hs = systems
    b = np.concatenate([gs.uniform_rhs(m.rows, 10 * i + j) for i, m in enumerate(mats) for j in range(nrhs)])
    out = []
    for graph in (0, 1):
        for overlap in (0, 1, 2):
            o = gs.SolverOptions(tol=1e-9, precision=precision, flexible=precision, use_graph=graph, lanes=lanes,
                                 overlap_launch=overlap, pre_steps=2)
            x, st = gs.Batch(hs, nrhs, o, device=device).solve(b)
            assert all(s.status == gs.STATUS_CONVERGED for s in st)
            out.append((x, [s.iterations for s in st]))
    for x, it in out[1:]:
        assert it == out[0][1] and np.array_equal(x, out[0][0])


@pytest.mark.parametrize("nrhs,precision", [(1, 0), (1, 1), (4, 0), (4, 1)])
@pytest.mark.parametrize("kw", [dict(), dict(omega=0.9), dict(pre_steps=2, post_steps=2), dict(coloring=1)],
                         ids=lambda kw: "-".join(f"{k}{v}" for k, v in kw.items()) or "default")
def test_cluster_steps_match_passes(gs, orc, device, nrhs, precision, kw):
    """The autotuned batch (one cluster per system and level where that is
    faster) against the colour passes alone (sweep_launch 0) and, in FP64, the
    oracle, on systems whose coarse levels have many small colours."""
    mats = [gs.varcoef_loguniform(x, y, z, seed=3 + i) for i, (x, y, z) in enumerate([(17, 19, 15), (21, 9, 23), (14, 14, 14)])]
    hs = [gs.Hierarchy.build(m, 1, 0.1, 10, 60) for m in mats]
    b = np.concatenate([gs.uniform_rhs(m.rows, 10 * i + j) for i, m in enumerate(mats) for j in range(nrhs)])
    out = []
    for sweep in (0, 1):
        for graph in (0, 1):
            o = gs.SolverOptions(tol=1e-9, precision=precision, flexible=precision, use_graph=graph, sweep_launch=sweep, **kw)
            B = gs.Batch(hs, nrhs, o, device=device)
            x, st = B.solve(b)
            assert all(s.status == gs.STATUS_CONVERGED for s in st)
            assert np.array_equal(B.solve(b)[0], x)
            out.append((x, [s.iterations for s in st]))
    # tol 1e-9 stops within one iteration whatever the rounding of an FP32 V-cycle
    bound = 1e-10 if precision == 0 else 1e-6
    for x, it in out[1:]:
        assert max(abs(p - q) for p, q in zip(it, out[0][1])) <= 1
        assert np.linalg.norm(x - out[0][0]) <= bound * np.linalg.norm(out[0][0])
