"""Performance cases: the calls that programs built on the library spend their time in.

Five kinds of pass, each through the public Python binding:

solve    one AMG-preconditioned CG solve, `Solver.solve_device` (or `Solver.solve` on host arrays), of a
         7-point variable-coefficient Poisson ("grf": log-normal coefficients, correlation length 8 cells,
         the distribution of the P128 benchmark; "loguni": independent log-uniform cells, the distribution
         of the batched benchmark), a Kuhn-tetrahedra P1 Laplacian ("kuhn") or P1 elasticity with 3x3
         blocks ("elast"). preset "plain" is the default drop-in (FP64 V-cycle, eager launches, the
         reference's algorithm, host-built hierarchy), "fast" the FP32 V-cycle inside an FP64 flexible CG
         with every fast option of the benchmark (GPU-built hierarchy).
batch    one `Batch.solve_device` of many uneven systems with 1 to 4 right-hand sides.
apply    one `Solver.apply_preconditioner_device` of the drop-in, for callers with an FP64 Krylov loop of
         their own.
backend  one smoothing-and-residual step written against the kernel-level Backend operations: a symmetric
         multicolour Gauss-Seidel step from zero, the product A x, the residual and its norm.

Plain solves stop at 1e-8 (the benchmark's tolerance), the mixed-precision ones at 1e-10, so that
the answers of two builds can be compared beyond the rounding of their FP32 V-cycles.
Matrices and right-hand sides are made here, from the seed, with torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-conjugate-gradient-solver_b200"))
import gpusolver_b200 as gs  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest single solve of the tests and of the benchmark (32^3), host arrays in and out:
        # launches and host round trips
        {"name": "poisson16_plain_host", "kind": "solve", "pde": "loguni", "nx": 16, "ny": 16, "nz": 16,
         "preset": "plain", "host": True},
        {"name": "poisson32_fast", "kind": "solve", "pde": "grf", "nx": 32, "ny": 32, "nz": 32, "preset": "fast",
         "host": False},
        # an ordinary drop-in solve on an odd box
        {"name": "poisson_61x47x83_plain", "kind": "solve", "pde": "loguni", "nx": 61, "ny": 47, "nz": 83,
         "preset": "plain", "host": False},
        # the headline workload
        {"name": "poisson128_fast", "kind": "solve", "pde": "grf", "nx": 128, "ny": 128, "nz": 128, "preset": "fast",
         "host": False},
        # unstructured-mesh Laplacian: 15 entries a row, more colours
        {"name": "kuhn64_fast", "kind": "solve", "pde": "kuhn", "m": 64, "preset": "fast", "host": False},
        {"name": "kuhn33_plain", "kind": "solve", "pde": "kuhn", "m": 33, "preset": "plain", "host": False},
        # elasticity, 3x3 block Gauss-Seidel
        {"name": "elast40_fast", "kind": "solve", "pde": "elast", "m": 40, "preset": "fast", "host": False},
        {"name": "elast17_plain", "kind": "solve", "pde": "elast", "m": 17, "preset": "plain", "host": False},
        # many uneven systems at once, four right-hand sides each
        {"name": "batch12_fast", "kind": "batch", "count": 12, "lo": 16, "hi": 56, "nrhs": 4, "preset": "fast"},
        # few small systems, one right-hand side, FP64
        {"name": "batch5_plain", "kind": "batch", "count": 5, "lo": 14, "hi": 30, "nrhs": 1, "preset": "plain"},
        # one V-cycle of the drop-in inside a caller's own Krylov loop
        {"name": "apply_72x65x58_plain", "kind": "apply", "pde": "grf", "nx": 72, "ny": 65, "nz": 58,
         "preset": "plain"},
        # unfused Backend operations in FP32 (the reference's arithmetic)
        {"name": "backend_kuhn48_f32", "kind": "backend", "pde": "kuhn", "m": 48, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["solve", "batch", "apply", "backend"], [8, 3, 2, 2])[0]
    if kind == "batch":
        lo = rng.randint(14, 24)
        preset = rng.choice(["plain", "fast"])
        return {"kind": kind, "count": rng.randint(3, 12), "lo": lo, "hi": lo + rng.randint(0, 30 if preset == "fast" else 12),
                "nrhs": rng.randint(1, 4), "preset": preset}
    preset = "plain" if kind == "apply" else rng.choice(["plain", "fast"])
    pde = rng.choices(["grf", "loguni", "kuhn", "elast"], [3, 2, 2, 2])[0]
    case = {"kind": kind, "pde": pde}
    if pde == "kuhn":
        case["m"] = _log(rng, 14, 64 if preset == "fast" else 40)
    elif pde == "elast":
        case["m"] = _log(rng, 10, 36 if preset == "fast" else 20)
    else:
        top = 96 if preset == "fast" else 64
        case.update(nx=_log(rng, 15, top), ny=_log(rng, 15, top), nz=_log(rng, 15, top))
    if kind == "backend":
        case["dtype"] = rng.choice(["f32", "f64"])
    else:
        case["preset"] = preset
    if kind == "solve":
        case["host"] = rng.random() < 0.25
    return case


# ---- matrices -----------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _poisson(pde, nx, ny, nz, g):
    """7-point finite volumes on nx x ny x nz cells, harmonic face means, zero Dirichlet values outside."""
    shape = (nz, ny, nx)
    f64 = dict(device=DEV, dtype=torch.float64)
    if pde == "grf":
        # exp(2.3 f), f white noise under a periodic Gaussian filter of 8 / sqrt(2) cells, standardised
        f = torch.fft.fftn(torch.randn(shape, generator=g, **f64))
        for d, n in enumerate(shape):
            k = torch.fft.fftfreq(n, **f64) * (2 * math.pi)
            f = f * torch.exp(-0.5 * (k * 8.0 / math.sqrt(2.0)) ** 2).reshape([-1 if e == d else 1 for e in range(3)])
        f = torch.fft.ifftn(f).real
        coef = torch.exp(2.3 * (f - f.mean()) / f.std())
    else:
        coef = torch.exp(math.log(0.1) + (math.log(10.0) - math.log(0.1)) * torch.rand(shape, generator=g, **f64))
    n = nx * ny * nz
    idx = torch.arange(n, device=DEV).reshape(shape)
    diag = torch.zeros(shape, **f64)
    cols, vals, keep = [None] * 7, [None] * 7, [None] * 7
    for d, step in ((0, nx * ny), (1, nx), (2, 1)):
        a, b = coef.narrow(d, 0, shape[d] - 1), coef.narrow(d, 1, shape[d] - 1)
        face = 2.0 * a * b / (a + b)
        for sign in (-1, 1):
            t = torch.zeros(shape, **f64)
            t.narrow(d, 1 if sign < 0 else 0, shape[d] - 1).copy_(face)
            inside = torch.zeros(shape, device=DEV, dtype=torch.bool)
            inside.narrow(d, 1 if sign < 0 else 0, shape[d] - 1).fill_(True)
            slot = d if sign < 0 else 6 - d
            cols[slot], vals[slot], keep[slot] = idx + sign * step, -t, inside
            diag += torch.where(inside, t, 2.0 * coef)
    cols[3], vals[3], keep[3] = idx, diag, torch.ones(shape, device=DEV, dtype=torch.bool)
    cols, vals, keep = (torch.stack([t.reshape(-1) for t in v], 1) for v in (cols, vals, keep))
    rp = torch.zeros(n + 1, device=DEV, dtype=torch.int64)
    rp[1:] = torch.cumsum(keep.sum(1), 0)
    return n, rp, cols[keep], vals[keep], None


def _tetrahedra(v):
    """The six Kuhn tetrahedra of every cube of a grid of v^3 vertices: (cells * 6, 4) vertex indices."""
    step = torch.tensor([1, v, v * v])
    paths = [[0, 1, 2], [0, 2, 1], [1, 0, 2], [1, 2, 0], [2, 0, 1], [2, 1, 0]]
    local = torch.stack([torch.cumsum(torch.cat([torch.zeros(1, dtype=torch.int64), step[p]]), 0) for p in paths])
    c = torch.arange(v - 1)
    base = (c[:, None, None] * v * v + c[None, :, None] * v + c[None, None, :]).reshape(-1)
    return (base[:, None, None] + local[None]).reshape(-1, 4).to(DEV)


def _gradients(x, t):
    """Volumes and gradients of the four linear basis functions of each tetrahedron."""
    p = x[t]
    e = p[:, 1:] - p[:, :1]
    inv = torch.linalg.inv(e)
    grad = inv.transpose(1, 2)
    grad = torch.cat([-grad.sum(1, keepdim=True), grad], 1)
    return torch.linalg.det(e).abs() / 6.0, grad


def _coo_to_csr(n, rows, cols, vals):
    m = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce()
    i = m.indices()
    rp = torch.zeros(n + 1, device=DEV, dtype=torch.int64)
    rp[1:] = torch.cumsum(torch.bincount(i[0], minlength=n), 0)
    return rp, i[1], m.values()


def _grid(v):
    c = torch.arange(v, device=DEV, dtype=torch.float64) / (v - 1)
    z, y, x = torch.meshgrid(c, c, c, indexing="ij")
    return torch.stack([x, y, z], -1).reshape(-1, 3)


def _kuhn(m, g):
    """P1 Laplacian on m^3 cubes of six tetrahedra, interior vertices moved by up to 0.2 of a cell."""
    v = m + 1
    x = _grid(v)
    at = torch.arange(v, device=DEV)
    inner = (at > 0) & (at < m)
    inner = (inner[:, None, None] & inner[None, :, None] & inner[None, None, :]).reshape(-1)
    move = (torch.rand(v ** 3, 3, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * (0.2 / m)
    x = torch.where(inner[:, None], x + move, x)
    t = _tetrahedra(v)
    vol, grad = _gradients(x, t)
    k = vol[:, None, None] * (grad @ grad.transpose(1, 2))
    number = torch.cumsum(inner.long(), 0) - 1
    rows, cols = t[:, :, None].expand(-1, 4, 4), t[:, None, :].expand(-1, 4, 4)
    keep = inner[rows] & inner[cols]
    n = int(inner.sum())
    return (n,) + _coo_to_csr(n, number[rows[keep]], number[cols[keep]], k[keep]) + (None,)


def _elasticity(v, g):
    """P1 elasticity on v^3 vertices, Young's modulus exp(N(0, 1)) per cube, Poisson ratio 0.3, the face
    x = 0 clamped, unit body force along -z; three interleaved unknowns a vertex."""
    x = _grid(v)
    t = _tetrahedra(v)
    vol, grad = _gradients(x, t)
    young = torch.exp(torch.randn((v - 1) ** 3, generator=g, device=DEV, dtype=torch.float64)).repeat_interleave(6)
    lam, mu = young * 0.3 / (1.3 * 0.4), young / 2.6
    free = x[:, 0] > 0
    number = torch.cumsum(free.long(), 0) - 1
    n = 3 * int(free.sum())
    rows, cols = t[:, :, None].expand(-1, 4, 4), t[:, None, :].expand(-1, 4, 4)
    keep = free[rows] & free[cols]
    ri, ci, parts = 3 * number[rows[keep]], 3 * number[cols[keep]], []
    dot = grad @ grad.transpose(1, 2)
    for a in range(3):
        for b in range(3):
            ga, gb = grad[:, :, a], grad[:, :, b]
            k = lam[:, None, None] * (ga[:, :, None] * gb[:, None, :]) + mu[:, None, None] * (gb[:, :, None] * ga[:, None, :])
            if a == b:
                k = k + mu[:, None, None] * dot
            parts.append((ri + a, ci + b, (vol[:, None, None] * k)[keep]))
    rp, col, val = _coo_to_csr(n, *(torch.cat(p) for p in zip(*parts)))
    load = torch.zeros(v ** 3, device=DEV, dtype=torch.float64)
    load.index_add_(0, t.reshape(-1), (vol / 4.0).repeat_interleave(4))
    rhs = torch.zeros(n, device=DEV, dtype=torch.float64)
    rhs[2::3] = -load[free]
    return n, rp, col, val, rhs


def _system(case, seed):
    """(n, row pointers, columns, values, right-hand side) on the GPU, FP64."""
    g = _generator(seed)
    if case["pde"] == "kuhn":
        n, rp, col, val, rhs = _kuhn(case["m"], g)
    elif case["pde"] == "elast":
        n, rp, col, val, rhs = _elasticity(case["m"], g)
    else:
        n, rp, col, val, rhs = _poisson(case["pde"], case["nx"], case["ny"], case["nz"], g)
    if rhs is None:
        rhs = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    return n, rp, col, val, rhs


def _batch_sides(case):
    """Sides spread evenly over [lo, hi], uneven ones among them; the same for every seed."""
    k = max(1, case["count"] - 1)
    return [case["lo"] + (case["hi"] - case["lo"]) * i // k for i in range(case["count"])]


def _batch_systems(case, seed):
    g = _generator(seed)
    out = []
    for side in _batch_sides(case):
        n, rp, col, val, _ = _poisson("loguni", side, side, side, g)
        out.append((n, rp, col, val, torch.rand(case["nrhs"], n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1))
    return out


def _csr(n, rp, col, val):
    return gs.Csr(n, n, rp.cpu().numpy().astype(np.int32), col.cpu().numpy().astype(np.int32), val.cpu().numpy())


# ---- plans --------------------------------------------------------------------
def _options(preset, block):
    # the cluster-resident coarse tail is off: its launch limit is one per process, and a program that
    # holds solvers of several systems at once (as this one does) cannot rely on it
    smoother = 1 if block == 3 else 0
    if preset == "plain":
        return gs.SolverOptions(smoother=smoother, tol=1e-8, max_iter=1000, coarse_solver=1, coarse_tail=0)
    return gs.SolverOptions(smoother=smoother, tol=1e-10, max_iter=1000, coarse_solver=1, precision=1, flexible=1,
                            use_graph=1, coarse_rows=24576, coloring=2, half_sweeps=1, coarse_half=1)


def _solver(case, a):
    block = 3 if case["pde"] == "elast" else 1
    if case["preset"] == "plain":
        h = gs.Hierarchy.build(a, block, 0.1, 10, 1000)
    else:
        h = gs.Hierarchy.build_ex(a, block, 0.1, 10, 1000, aggregation=1, device=0)
    return gs.Solver(h, _options(case["preset"], block), device=0)


def prepare(case, seed):
    torch.cuda.set_device(0)
    kind = case["kind"]
    if kind == "batch":
        systems = _batch_systems(case, seed)
        hs = [gs.Hierarchy.build(_csr(*s[:4]), 1, 0.1, 10, 1000) for s in systems]
        if case["preset"] == "plain":
            opts = gs.SolverOptions(tol=1e-8, max_iter=1000, coarse_solver=1)
        else:
            opts = gs.SolverOptions(tol=1e-10, max_iter=1000, coarse_solver=1, precision=1, flexible=1, use_graph=1,
                                    coarse_rows=4096, coloring=1)
        b = torch.cat([s[4].reshape(-1) for s in systems])
        return {"kind": kind, "batch": gs.Batch(hs, case["nrhs"], opts, device=0), "b": b, "x": torch.zeros_like(b)}
    n, rp, col, val, rhs = _system(case, seed)
    if kind == "backend":
        return _prepare_backend(case, n, rp, col, val, rhs)
    s = _solver(case, _csr(n, rp, col, val))
    if case.get("host"):
        return {"kind": "host", "solver": s, "b": rhs.cpu().numpy()}
    return {"kind": kind, "solver": s, "b": rhs, "x": torch.zeros_like(rhs)}


def _node_graph(a, block):
    """Pattern that the colouring walks: the matrix itself, or its graph of 3x3 blocks."""
    if block == 1:
        return a
    rp, col = gs.block_graph(a, 3)
    return gs.Csr(a.rows // 3, a.rows // 3, rp, col, np.ones(len(col)))


def _prepare_backend(case, n, rp, col, val, rhs):
    block = 3 if case["pde"] == "elast" else 1
    dt, code = (torch.float32, gs.F32) if case["dtype"] == "f32" else (torch.float64, gs.F64)
    a = _csr(n, rp, col, val)
    _, _, verts, offs = gs.greedy_coloring(_node_graph(a, block))
    s = {"kind": "backend", "A": gs.DeviceCsr(a, code), "code": code, "n": n, "block": block,
         "order": torch.from_numpy(verts).to(DEV), "offs": [int(o) for o in offs], "b": rhs.to(dt)}
    if block == 3:
        s["dinv"] = torch.from_numpy(gs.block_inverses3x3(a)).to(DEV).to(dt)
    s.update(x=torch.zeros_like(s["b"]), y=torch.zeros_like(s["b"]), r=torch.zeros_like(s["b"]),
             rr=torch.zeros(1, device=DEV, dtype=dt))
    return s


# ---- one pass -----------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "host":
        return state["solver"].solve(state["b"])[0]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "backend":
        return _run_backend(state, stream)
    b, x = state["b"], state["x"]
    if kind == "apply":
        state["solver"].apply_preconditioner_device(b.data_ptr(), x.data_ptr(), stream)
        return x
    x.zero_()
    if kind == "batch":
        state["batch"].solve_device(b.data_ptr(), x.data_ptr(), stream)
    else:
        state["solver"].solve_device(b.data_ptr(), x.data_ptr(), stream)
    return x


def _run_backend(s, stream):
    n, code, order, offs = s["n"], s["code"], s["order"].data_ptr(), s["offs"]
    b, x, y, r, rr = (s[k].data_ptr() for k in ("b", "x", "y", "r", "rr"))
    gs.vector_op(gs.VEC_SET_ZERO, n, x, x, dtype=code, stream=stream)
    colours = list(range(len(offs) - 1))
    for c in colours + colours[::-1]:
        if s["block"] == 3:
            gs.block_gauss_seidel_color3x3(s["A"], order, offs[c], offs[c + 1] - offs[c], s["dinv"].data_ptr(), b, x, 1.0,
                                           stream)
        else:
            gs.gauss_seidel_color(s["A"], order, offs[c], offs[c + 1] - offs[c], b, x, 1.0, stream)
    gs.spmv(s["A"], x, y, stream)
    gs.vector_op(gs.VEC_COPY, n, b, r, dtype=code, stream=stream)
    gs.vector_op(gs.VEC_AXPY, n, y, r, alpha=-1.0, dtype=code, stream=stream)
    gs.dot(n, r, r, rr, code, stream)
    return {"x": s["x"], "r": s["r"], "rr": s["rr"]}


# ---- what a pass cannot do without ----------------------------------------------
def _sizes(case):
    """(unknowns, stored entries) of a case's matrix."""
    if case["pde"] == "kuhn":
        w = v = case["m"] - 1
    elif case["pde"] == "elast":
        v = case["m"]
        w = v - 1
    if case["pde"] in ("kuhn", "elast"):
        # a vertex couples to itself and along +-(edge, face diagonal, body diagonal): 15 at most
        edges = (w - 1) * v * v + 2 * w * (v - 1) * v + 2 * (w - 1) * (v - 1) * v + w * (v - 1) ** 2 + (w - 1) * (v - 1) ** 2
        b = 3 if case["pde"] == "elast" else 1
        return b * w * v * v, b * b * (w * v * v + 2 * edges)
    x, y, z = case["nx"], case["ny"], case["nz"]
    return x * y * z, 7 * x * y * z - 2 * (x * y + y * z + x * z)


def work(case):
    """The matrix, the right-hand side and the answer once each; a solve cannot do without one product per
    iteration either, but how many it takes is the method's, so a pass counts one."""
    if case["kind"] == "batch":
        sizes = [(s ** 3, 7 * s ** 3 - 6 * s * s) for s in _batch_sides(case)]
        n, nnz, r = sum(s[0] for s in sizes), sum(s[1] for s in sizes), case["nrhs"]
        return {"bytes": 12 * nnz + 4 * n + 16 * n * r, "flops": 2 * nnz * r}
    n, nnz = _sizes(case)
    size = 4 if case.get("dtype") == "f32" else 8
    products = 3 if case["kind"] == "backend" else 1
    vectors = 4 if case["kind"] == "backend" else 2
    return {"bytes": (4 + size) * nnz + 4 * n + size * vectors * n, "flops": 2 * nnz * products}


# ---- the same in 64 bits, plain torch ---------------------------------------------
def _pcg(a, diag, b):
    """Jacobi-preconditioned CG to the end of FP64's accuracy, restarted from the true residual."""
    x = torch.zeros_like(b)
    target = 1e-14 * float(torch.linalg.vector_norm(b))
    for _ in range(4):
        r = b - a @ x
        z = r / diag
        p, rz = z.clone(), torch.dot(r, z)
        goal = max(target, 1e-11 * float(torch.linalg.vector_norm(r)))
        for it in range(20000):
            ap = a @ p
            alpha = rz / torch.dot(p, ap)
            x += alpha * p
            r -= alpha * ap
            if it % 25 == 24 and float(torch.linalg.vector_norm(r)) < goal:
                break
            z = r / diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        if float(torch.linalg.vector_norm(b - a @ x)) < 4 * target:
            break
    return x


def _torch_csr(n, rp, col, val):
    a = torch.sparse_csr_tensor(rp, col, val, (n, n))
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    return a, val[rows == col], rows


def exact(case, seed):
    if case["kind"] == "apply":
        return None
    if case["kind"] == "batch":
        systems = _batch_systems(case, seed)
        out = []
        for n, rp, col, val, rhs in systems:
            a, diag, _ = _torch_csr(n, rp, col, val)
            out += [_pcg(a, diag, r) for r in rhs]
        return torch.cat(out)
    n, rp, col, val, rhs = _system(case, seed)
    a, diag, rows = _torch_csr(n, rp, col, val)
    if case["kind"] == "solve":
        return _pcg(a, diag, rhs)
    # the Backend step on the values and the right-hand side as the step is given them
    block = 3 if case["pde"] == "elast" else 1
    if case["dtype"] == "f32":
        val, rhs = val.float().double(), rhs.float().double()
        a, diag, rows = _torch_csr(n, rp, col, val)
    _, _, verts, offs = gs.greedy_coloring(_node_graph(_csr(n, rp, col, val), block))
    verts = torch.from_numpy(verts).to(DEV).long()
    x = torch.zeros_like(rhs)
    blocks = torch.zeros(n // block, block, block, device=DEV, dtype=torch.float64)
    inside = rows // block == col // block
    blocks[rows[inside] // block, rows[inside] % block, col[inside] % block] = val[inside]
    inv = torch.linalg.inv(blocks)
    colours = list(range(len(offs) - 1))
    for c in colours + colours[::-1]:
        nodes = verts[int(offs[c]):int(offs[c + 1])]
        res = (rhs - a @ x).reshape(-1, block)[nodes]
        x.reshape(-1, block)[nodes] += (inv[nodes] @ res[:, :, None])[:, :, 0]
    r = rhs - a @ x
    return {"x": x, "r": r, "rr": torch.dot(r, r).reshape(1)}
