"""Performance cases of the sparse Cholesky path, through its public Python entry points.

A case names a matrix family and size, a number of right-hand sides and a call:

* ``step``: NumericFactorization of new values and Solve on CUDA tensors, the symbolic analysis
  held (a time step, a Newton step, a new set of coefficients on an old mesh);
* ``host_step``: the same from host arrays to a host array;
* ``solve``: Solve on CUDA tensors with a factor held;
* ``cg``: ConjugateGradient on a nearby matrix, preconditioned by a factor held;
* ``batch``: BatchedCholesky over many independent meshes, NumericFactorization and Solve.

The families are the benchmark's and the tests' own: 2D 5-point grids, 2D quality meshes
(triangulated jittered grids), 3D 7-point grids, and the 3-dof 27-point vector Laplacian, all with
random positive coefficients.  Coefficients, shift and solution are rounded to dyadic grids coarse
enough that B = (A + shift I) X is formed without any rounding, so X is the exact solution.
"""
import functools

import numpy as np
import torch

from tensors_b200 import matrices, ordering
from tensors_b200.cholesky import BatchedCholesky, CholeskyDecomposition

COEF_STEP = 2.0 ** -20     # coefficients are multiples of it
SOL_STEP = 2.0 ** -14      # solutions are multiples of it
SHIFT = 2.0 ** -7          # the tests' and the serving workload's diagonal shift, 1e-2
SMALL_SHIFT = 2.0 ** -20   # the headline 3D grid's, 1e-6


def listed():
    return [
        # the smallest call: one right-hand side against a held factor, all launches and latency
        dict(name="solve_grid2d_32_k1", kind="grid2d", size=32, k=1, call="solve", precision="fp64", shift=SHIFT),
        # a small odd-sized refactorization in somebody's inner loop
        dict(name="step_grid2d_45_k4", kind="grid2d", size=45, k=4, call="step", precision="fp64", shift=SHIFT),
        # a mid-sized mesh driven from host arrays, as code without torch does
        dict(name="host_step_mesh2d_131_k2", kind="mesh2d", size=131, k=2, call="host_step", precision="fp64", shift=SHIFT),
        # the serving workload's largest mesh, mixed precision refined to 1e-10
        dict(name="step_mesh2d_224_k16_mixed", kind="mesh2d", size=224, k=16, call="step", precision="mixed", tol=1e-10,
             shift=SHIFT),
        # a ragged 3D grid, one right-hand side, FP64
        dict(name="step_grid3d_31_k1", kind="grid3d", size=31, k=1, call="step", precision="fp64", shift=SHIFT),
        # the serving workload's 3D grid, mixed precision refined to 1e-10
        dict(name="step_grid3d_48_k8_mixed", kind="grid3d", size=48, k=8, call="step", precision="mixed", tol=1e-10,
             shift=SHIFT),
        # the headline workload: FP64 factor + solve of the 64^3 grid with 16 right-hand sides
        dict(name="step_grid3d_64_k16", kind="grid3d", size=64, k=16, call="step", precision="fp64", shift=SMALL_SHIFT),
        # repeated solves with the widest right-hand-side block of the serving workload
        dict(name="solve_grid3d_56_k64", kind="grid3d", size=56, k=64, call="solve", precision="fp64", shift=SHIFT),
        # a factor kept for a few time steps: conjugate gradients on the changed matrix
        dict(name="cg_grid3d_40_k4", kind="grid3d", size=40, k=4, call="cg", precision="fp64", shift=SHIFT),
        # many independent meshes of different sizes in one call
        dict(name="batch_96_meshes", kind="batch", size=100, count=96, k=1, call="batch", precision="fp64", shift=SHIFT),
        # the 3-dof vector Laplacian with direct FP64 solves
        dict(name="step_vector3d_33_k8", kind="vector3d", size=33, k=8, call="step", precision="fp64", shift=SHIFT),
        # the mixed-precision headline: its full 48^3 size, refined to 1e-12
        dict(name="step_vector3d_48_k8_mixed", kind="vector3d", size=48, k=8, call="step", precision="mixed", tol=1e-12,
             shift=SHIFT),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["grid2d", "mesh2d", "grid3d", "grid3d", "vector3d", "batch"])
    if kind == "batch":
        return dict(kind=kind, size=log_int(24, 100), count=log_int(6, 120), k=1, call="batch", precision="fp64", shift=SHIFT)
    lo, hi = dict(grid2d=(20, 240), mesh2d=(24, 224), grid3d=(9, 60), vector3d=(6, 36))[kind]
    case = dict(kind=kind, size=log_int(lo, hi), k=log_int(1, 64), call=rng.choice(["step", "step", "solve", "solve", "host_step", "cg"]),
                precision="fp64", shift=SHIFT)
    if case["call"] != "cg" and rng.random() < 0.4:
        case.update(precision="mixed", tol=rng.choice([1e-10, 1e-12]))
    return case


# ------------------------------------------------------------------ patterns
class Pattern:
    """A symmetric block pattern with the diagonal, its fill-reducing order, and where each edge's
    blocks lie in the CSR value array."""

    def __init__(self, nodes, a, b, weight, dofs, perm_nodes):
        d = self.dofs = dofs
        self.nodes, self.n, self.edges = nodes, nodes * dofs, len(a)
        rows = np.concatenate([a, b, np.arange(nodes)])
        cols = np.concatenate([b, a, np.arange(nodes)])
        order = np.argsort(rows * nodes + cols, kind="stable")
        slot = np.empty(len(rows), dtype=np.int64)
        slot[order] = np.arange(len(rows))
        count = np.bincount(rows, minlength=nodes)
        start = np.concatenate([[0], np.cumsum(count)])
        self.nnz = len(rows) * d * d
        # dof row d p + i holds the d columns of each of node p's neighbours in order
        i, j = np.arange(d)[None, :, None], np.arange(d)[None, None, :]
        base = start[rows] * d * d + (slot - start[rows]) * d
        where = base[:, None, None] + i * (count[rows] * d)[:, None, None] + j
        e = len(a)
        self.at_ab, self.at_ba, self.at_diag = where[:e], where[e:2 * e], where[2 * e:]
        self.a, self.b, self.weight = a, b, weight
        row_len = np.repeat(count * d, d)
        self.outer = np.concatenate([[0], np.cumsum(row_len)]).astype(np.int64)
        inner = np.empty(self.nnz, dtype=np.int32)
        inner[where] = (cols * d)[:, None, None] + np.broadcast_to(j, where.shape)
        self.inner = inner
        self.perm = (perm_nodes[:, None].astype(np.int64) * d + np.arange(d)).ravel().astype(np.int32)


def _grid_edges(size, dim, offsets):
    idx = np.arange(size ** dim, dtype=np.int64).reshape((size,) * dim)
    a, b = [], []
    for off in offsets:
        lo = tuple(slice(max(0, -o), size - max(0, o)) for o in off)
        hi = tuple(slice(max(0, o), size - max(0, -o)) for o in off)
        a.append(idx[lo].ravel())
        b.append(idx[hi].ravel())
    return np.concatenate(a), np.concatenate(b)


def _node_matrix(nodes, a, b, coords):
    rows = np.concatenate([a, b, np.arange(nodes)])
    cols = np.concatenate([b, a, np.arange(nodes)])
    key = np.sort(rows * nodes + cols)
    outer = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nodes))]).astype(np.int64)
    return matrices.CSRMatrix(n=nodes, outer=outer, inner=(key % nodes).astype(np.int32), values=np.ones(len(key)), coords=coords)


@functools.lru_cache(maxsize=None)
def _pattern(kind, size):
    if kind == "mesh2d":
        A = matrices.mesh_laplacian(size * size, size, 1e-2, relative=True)
        rows = np.repeat(np.arange(A.n, dtype=np.int64), np.diff(A.outer))
        up = rows < A.inner
        weight = np.maximum(np.abs(A.values[up]), 2.0 ** -6)     # positive: definite for any coefficients
        return Pattern(A.n, rows[up], A.inner[up].astype(np.int64), weight, 1, ordering.nested_dissection(A))
    if kind == "grid2d":
        a, b = _grid_edges(size, 2, [(0, 1), (1, 0)])
        return Pattern(size ** 2, a, b, np.ones(len(a)), 1, ordering.nested_dissection(_node_matrix(size ** 2, a, b, None)))
    if kind == "grid3d":
        # the pattern-only dissection: half the coordinate one's factor flops on these grids
        a, b = _grid_edges(size, 3, [(1, 0, 0), (0, 1, 0), (0, 0, 1)])
        return Pattern(size ** 3, a, b, np.ones(len(a)), 1, ordering.nested_dissection(_node_matrix(size ** 3, a, b, None)))
    offsets = [(z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1) if (z, y, x) > (0, 0, 0)]
    a, b = _grid_edges(size, 3, offsets)
    coords = np.stack(np.meshgrid(*[np.arange(size)] * 3, indexing="ij"), axis=-1).reshape(-1, 3).astype(np.float64)
    return Pattern(size ** 3, a, b, np.ones(len(a)), 3, ordering.nested_dissection(_node_matrix(size ** 3, a, b, coords)))


def _batch_sizes(case):
    # mesh edges from a quarter of `size` to `size`, repeatedly, in an order without runs
    lo, hi, count = max(6, case["size"] // 4), case["size"], case["count"]
    return [lo + (7919 * s) % (hi - lo + 1) for s in range(count)]


def _patterns(case):
    if case["call"] == "batch":
        return [_pattern("mesh2d", g) for g in _batch_sizes(case)]
    return [_pattern(case["kind"], case["size"])]


# -------------------------------------------------------------------- inputs
def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 4 + stream)


def _round(x, step):
    return torch.round(x / step) * step


def _on_gpu(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _coefficients(p, gen):
    """Positive edge coefficients: weight * lognormal, or SPD 3 x 3 blocks G G^T + 0.1 I."""
    if p.dofs == 1:
        w = _on_gpu(p.weight) * torch.exp(torch.randn(p.edges, dtype=torch.float64, device="cuda", generator=gen))
        return torch.clamp(_round(w, COEF_STEP), min=COEF_STEP).reshape(-1, 1, 1)
    G = torch.randn(p.edges, 3, 3, dtype=torch.float64, device="cuda", generator=gen)
    W = G @ G.transpose(1, 2) + 0.1 * torch.eye(3, dtype=torch.float64, device="cuda")
    return _round(0.5 * (W + W.transpose(1, 2)), COEF_STEP)


def _values(p, W):
    """CSR values of sum_e [[W, -W], [-W, W]] (sums of multiples of COEF_STEP: exact)."""
    vals = torch.empty(p.nnz, dtype=torch.float64, device="cuda")
    vals[_on_gpu(p.at_ab).reshape(-1)] = -W.reshape(-1)
    vals[_on_gpu(p.at_ba).reshape(-1)] = -W.reshape(-1)
    diag = torch.zeros(p.nodes, p.dofs, p.dofs, dtype=torch.float64, device="cuda")
    diag.index_add_(0, _on_gpu(p.a), W)
    diag.index_add_(0, _on_gpu(p.b), W)
    vals[_on_gpu(p.at_diag).reshape(-1)] = diag.reshape(-1)
    return vals


def _solution(n, k, seed):
    X = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=_generator(seed, 1))
    return torch.clamp(_round(X, SOL_STEP), -6.0, 6.0)


def _shape(case, X):
    return X.reshape(-1) if case["k"] == 1 else X


def _right_hand_side(ps, values, X, shift):
    parts, row = [], 0
    for p, v in zip(ps, values):
        A = torch.sparse_csr_tensor(_on_gpu(p.outer), _on_gpu(p.inner.astype(np.int64)), v, size=(p.n, p.n))
        x = X[row:row + p.n].contiguous()
        parts.append(A @ x + shift * x)
        row += p.n
    return torch.cat(parts)


@functools.lru_cache(maxsize=None)
def _stream():
    """The program's working stream; every handle runs on it."""
    return torch.cuda.Stream()


def prepare(case, seed):
    ps = _patterns(case)
    n, k, gen = sum(p.n for p in ps), case["k"], _generator(seed, 0)
    coefs = [_coefficients(p, gen) for p in ps]
    values = [_values(p, W) for p, W in zip(ps, coefs)]
    if case["call"] == "batch":
        solver = BatchedCholesky([(p.outer, p.inner, p.perm) for p in ps])
        handle = solver.handle
    else:
        solver = handle = CholeskyDecomposition(ps[0].outer, ps[0].inner, ps[0].perm)
    handle.SetPrecision(case["precision"])
    if case["precision"] == "mixed":
        handle.SetRefinement(case["tol"], 30)
    handle.SetStream(_stream())
    handle.SymbolicFactorization()
    state = dict(case=case, solver=solver)
    if case["call"] in ("solve", "cg"):
        torch.cuda.synchronize()
        assert solver.NumericFactorization(torch.cat(values), case["shift"]) == 0
    if case["call"] == "cg":
        # the matrix has moved on since the factorization: coefficients changed by up to a tenth
        change = 1.0 + 0.1 * (2.0 * torch.rand(coefs[0].shape[0], 1, 1, dtype=torch.float64, device="cuda", generator=gen) - 1.0)
        values = [_values(ps[0], torch.clamp(_round(coefs[0] * change, COEF_STEP), min=COEF_STEP) if ps[0].dofs == 1
                          else _round(coefs[0] * change, COEF_STEP))]
    B = _shape(case, _right_hand_side(ps, values, _solution(n, k, seed), case["shift"]))
    state.update(values=torch.cat(values), B=B, X=torch.empty_like(B))
    if case["call"] == "host_step":
        state.update(values=state["values"].cpu().numpy(), B=B.cpu().numpy(), X=np.zeros(B.shape))
    torch.cuda.synchronize()
    return state


def run(state):
    case, solver, X = state["case"], state["solver"], state["X"]
    with torch.cuda.stream(_stream()):
        if case["call"] == "cg":
            _, succeeded = solver.ConjugateGradient(state["B"], X, values=state["values"], reg=case["shift"],
                                                    relative_tolerance=1e-10, max_iter=100)
            assert succeeded
            return X
        if case["call"] != "solve":
            assert solver.NumericFactorization(state["values"], case["shift"]) == 0
        solver.Solve(state["B"], X)
    return X


# ---------------------------------------------------------------- references
@functools.lru_cache(maxsize=None)
def _factor_counts(kind, size):
    p = _pattern(kind, size)
    return CholeskyDecomposition(p.outer, p.inner, p.perm).FlopCount()


def work(case):
    """Values and right-hand sides in, solutions out, each once; a solve also reads the held factor
    (nonzeros of U) once.  Flops of the factorization and of two sweeps (one application for cg)."""
    kinds = [("mesh2d", g) for g in _batch_sizes(case)] if case["call"] == "batch" else [(case["kind"], case["size"])]
    counts = [_factor_counts(*q) for q in kinds]
    ps = _patterns(case)
    factor, nnz_u = sum(c[0] for c in counts), sum(c[1] for c in counts)
    n, nnz, k = sum(p.n for p in ps), sum(p.nnz for p in ps), case["k"]
    item = 4 if case["precision"] == "mixed" else 8
    bytes_ = 16.0 * n * k
    flops = 4.0 * k * nnz_u
    if case["call"] in ("solve", "cg"):
        bytes_ += item * nnz_u
    if case["call"] != "solve":
        bytes_ += 8.0 * nnz
    if case["call"] not in ("solve", "cg"):
        flops += factor
    return {"bytes": bytes_, "flops": flops}


def exact(case, seed):
    """The solution that the right-hand side was formed from, without rounding."""
    if case["call"] == "batch":
        n = sum(g * g for g in _batch_sizes(case))
    else:
        n = {"grid2d": case["size"] ** 2, "mesh2d": case["size"] ** 2, "grid3d": case["size"] ** 3, "vector3d": 3 * case["size"] ** 3}[case["kind"]]
    return _shape(case, _solution(n, case["k"], seed))
