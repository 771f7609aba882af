"""The calls of this framework whose speed is looked after.

A case is a dict of plain values; `prepare` makes what a program holds before the call (matrix, right-hand
side, solver), `run` makes the call through the public classes, `work` counts what the call cannot do
without, and `exact` computes the same result in 64 bits with plain torch: its own element matrices, its
own sparse matrix and its own conjugate gradients.

`call` of a case:
  product    CSROperator.product, the operator behind every solver (FP64 and FP32 spaces)
  cg         ConjugateGradients with makeDiagonalOperator, the drop-in solve (FP64)
  mixed      MixedPrecisionCG, the same solve with FP32 inner iterations
  batch      BatchedConjugateGradients over uneven systems (FP64, or FP32 with reliable updates)
  multi      MultiRHSConjugateGradients, several right-hand sides on one matrix (FP64, or FP32 refined)
  assemble   Assembler.assemble of a new coefficient field, then the Dirichlet elimination
  embedded   Assembler.assemble_embedded (finite cells, FP64 or the FP32 tensor-core copy) and elimination
  adjoint    DifferentiablePoisson, forward and backward for two coefficient fields in turn
  two_level  TwoLevelCG with FP32 smoothing on a finite-cell sphere
"""
import math
import random

import numpy as np
import torch

TOLERANCE = 1e-10  # relative residual of the solves, the one the benchmark asks for
ALPHA, RADIUS, DEPTH = 1e-6, 0.4, 2  # the finite-cell sphere of the benchmark


def listed():
    return [
        # A small operator product, as a host-driven iteration on a 2D Q1 mesh makes them by the thousand:
        # its time is the call and one launch.
        {"name": "product_2d_q1_64", "call": "product", "dim": 2, "order": 1, "nx": 64, "ny": 64, "dtype": "f64"},
        # The operator product of the benchmark's 3D matrix (57 million entries).
        {"name": "product_3d_q1_128", "call": "product", "dim": 3, "order": 1, "nx": 128, "ny": 128, "nz": 128,
         "dtype": "f64"},
        # The benchmark's small solve: 2D Q1 on 256 x 256 cells, the whole system on chip.
        {"name": "cg_2d_q1_256", "call": "cg", "dim": 2, "order": 1, "nx": 256, "ny": 256},
        # The benchmark's FP64 solve on 128^3 cells.
        {"name": "cg_3d_q1_128", "call": "cg", "dim": 3, "order": 1, "nx": 128, "ny": 128, "nz": 128},
        # A quadratic 3D mesh of odd size: a general sparse matrix (125 diagonals), solved in FP64.
        {"name": "cg_3d_q2_31", "call": "cg", "dim": 3, "order": 2, "nx": 31, "ny": 31, "nz": 31},
        # The benchmark's headline: the 128^3 solve with FP32 inner iterations and FP64 refinement.
        {"name": "mixed_3d_q1_128", "call": "mixed", "dim": 3, "order": 1, "nx": 128, "ny": 128, "nz": 128},
        # Parameter studies: many independent 2D Q2 systems of 16 .. 128 cells a side, solved together.
        {"name": "batch_64_q2", "call": "batch", "systems": 64, "smallest": 16, "largest": 128, "dtype": "f64"},
        # 32 load cases on the benchmark's 3D matrix, FP32 iterations refined in FP64.
        {"name": "multi_32_3d_q1_128", "call": "multi", "dim": 3, "order": 1, "nx": 128, "ny": 128, "nz": 128,
         "columns": 32, "dtype": "f32"},
        # A new coefficient field on a fixed mesh, as every step of a parameter study assembles it.
        {"name": "assemble_3d_q1_128", "call": "assemble", "dim": 3, "order": 1, "nx": 128, "ny": 128, "nz": 128},
        # The cubic finite-cell sphere of the benchmark, its FP64 matrix.
        {"name": "embedded_q3_32", "call": "embedded", "dim": 3, "order": 3, "nx": 32, "dtype": "f64"},
        # A step of an inverse problem on 64^3 cells: two fields, forward and backward each.
        {"name": "adjoint_3d_q1_64", "call": "adjoint", "dim": 3, "order": 1, "nx": 64, "ny": 64, "nz": 64},
        # The preconditioned solve of the finite-cell sphere at a quarter of the benchmark's unknowns and below.
        {"name": "two_level_q3_16", "call": "two_level", "dim": 3, "order": 3, "nx": 16},
    ]


def draw(rng):
    """A case of the same calls, its sizes spread over what the listed ones stand for."""

    def between(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def box(dim, a, b):
        n = between(a, b)
        side = {"nx": n, "ny": max(a // 2, int(n * rng.uniform(0.7, 1.0)))}
        if dim == 3:
            side["nz"] = max(a // 2, int(n * rng.uniform(0.7, 1.0)))
        return side

    call = rng.choice(["product", "cg", "mixed", "batch", "multi", "assemble", "embedded", "adjoint", "two_level"])
    if call == "product":
        dim, order = rng.choice([(2, 1), (2, 2), (3, 1), (3, 1), (3, 2), (3, 3)])
        a, b = {(2, 1): (40, 1200), (2, 2): (24, 600), (3, 1): (12, 128), (3, 2): (8, 44), (3, 3): (6, 24)}[dim, order]
        return {"call": call, "dim": dim, "order": order, **box(dim, a, b), "dtype": rng.choice(["f64", "f64", "f32"])}
    if call in ("cg", "mixed"):
        dim, order = rng.choice([(2, 1), (3, 1), (3, 1), (3, 2)])
        a, b = {(2, 1): (48, 700), (3, 1): (16, 128), (3, 2): (8, 36)}[dim, order]
        return {"call": call, "dim": dim, "order": order, **box(dim, a, b)}
    if call == "batch":
        return {"call": call, "systems": between(4, 64), "smallest": 16, "largest": rng.randint(48, 128),
                "dtype": rng.choice(["f64", "f32"])}
    if call == "multi":
        return {"call": call, "dim": 3, "order": 1, **box(3, 20, 110), "columns": rng.choice([2, 5, 8, 13, 16, 32, 32]),
                "dtype": rng.choice(["f64", "f32"])}
    if call == "assemble":
        dim, order = rng.choice([(2, 1), (2, 2), (3, 1), (3, 1), (3, 2), (3, 3)])
        a, b = {(2, 1): (64, 1000), (2, 2): (32, 400), (3, 1): (16, 128), (3, 2): (8, 44), (3, 3): (6, 24)}[dim, order]
        return {"call": call, "dim": dim, "order": order, **box(dim, a, b)}
    if call == "embedded":
        return {"call": call, "dim": 3, "order": rng.choice([2, 3]), "nx": between(8, 32),
                "dtype": rng.choice(["f64", "f32"])}
    if call == "adjoint":
        return {"call": call, "dim": 3, "order": 1, **box(3, 12, 72)}
    return {"call": call, "dim": 3, "order": 3, "nx": between(8, 16)}


# ---- the meshes and the seeded inputs ----------------------------------------------------------------

def _cells(case):
    if case["call"] in ("embedded", "two_level"):
        return [case["nx"]] * case["dim"]
    return [case[k] for k in ("nx", "ny", "nz")[: case["dim"]]]


def _sizes(case):
    """Systems of a batch: cells a side, the same for every seed."""
    rng = random.Random(7919 * case["systems"] + case["largest"])
    return [rng.randint(case["smallest"], case["largest"]) for _ in range(case["systems"])]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _kappa(cells, g):
    """exp of a unit-variance Gaussian field smoothed over three cells, first axis fastest."""
    f = torch.randn(tuple(reversed(cells)), generator=g, device="cuda", dtype=torch.float64)
    w = torch.exp(-0.5 * torch.arange(-3, 4, device="cuda", dtype=torch.float64) ** 2)
    w = w / w.sum()
    for d in range(f.dim()):
        n = f.shape[d]
        at = torch.arange(n, device="cuda")
        f = sum(w[j + 3] * f.index_select(d, (at + j).clamp(0, n - 1)) for j in range(-3, 4))
    return torch.exp((f - f.mean()) / f.std(unbiased=False)).reshape(-1)


def _uniform(n, g, columns=None):
    shape = (n,) if columns is None else (n, columns)
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * 2 - 1


def _inputs(case, seed):
    """(kappas, right-hand side) of a case, from the seed alone; `system` counts the systems of a batch."""
    g = _generator(seed)
    if case["call"] == "batch":
        out = []
        for n in _sizes(case):
            k = _kappa([n, n], g)
            out.append((k, _uniform((2 * n + 1) ** 2, g)))
        return out
    cells = _cells(case)
    n = math.prod(case["order"] * c + 1 for c in cells)
    count = 2 if case["call"] == "adjoint" else 0 if case["call"] in ("embedded", "two_level") else 1
    kappas = [_kappa(cells, g) for _ in range(count)]
    return kappas, _uniform(n, g, case.get("columns"))


def _tight():
    from cie_b200.linalg import Statistics
    return Statistics(20000, 0.0, TOLERANCE)


def _pattern(space, mesh):
    """An empty matrix in the pattern of the mesh and the boundary flags."""
    from cie_b200.graph import csr_pattern_device
    from cie_b200.linalg import CSRMatrix
    dofmap = torch.as_tensor(mesh.dofmap).to(space.device)
    rowptr, col = csr_pattern_device(space, mesh.ncells, mesh.nb, dofmap, mesh.ndofs)
    matrix = CSRMatrix(mesh.ndofs, rowptr, col, torch.zeros(col.numel(), dtype=torch.float64, device=space.device))
    return matrix, torch.as_tensor(mesh.boundary()).to(space.device), dofmap


def _system(space, dim, order, cells, kappa, rhs=None):
    """The assembled and eliminated matrix; rows of `rhs` on the boundary are zeroed."""
    from cie_b200.fem import Assembler, StructuredMesh
    mesh = StructuredMesh(dim, order, cells)
    matrix, boundary, dofmap = _pattern(space, mesh)
    assembler = Assembler(space, matrix, mesh, d_dofmap=dofmap)
    assembler.assemble(kappa)
    assembler.dirichlet(boundary, rhs)
    return mesh, matrix, boundary, assembler


def prepare(case, seed):
    from cie_b200.fem import Assembler, PoissonProblem, StructuredMesh
    from cie_b200.linalg import (BatchedConjugateGradients, ConjugateGradients, CSROperator, CUDASpace,
                                 MixedPrecisionCG, MultiRHSConjugateGradients, block_diagonal, makeDiagonalOperator)
    call = case["call"]
    space = CUDASpace()
    state = {"call": call, "space": space}

    if call == "batch":
        matrices, rhs = [], []
        for n, (kappa, b) in zip(_sizes(case), _inputs(case, seed)):
            matrices.append(_system(space, 2, 2, [n, n], kappa, b)[1])
            rhs.append(b)
        torch.cuda.synchronize()
        matrix, offsets = block_diagonal(matrices)
        solver = BatchedConjugateGradients(matrix, offsets, space, makeDiagonalOperator(matrix, space), _tight())
        if case["dtype"] == "f32":
            solver.set_reliable_updates(0.1)
        return dict(state, solver=solver, b=torch.cat(rhs))

    dim, order, cells = case["dim"], case["order"], _cells(case)
    kappas, b = _inputs(case, seed)

    if call == "adjoint":
        from cie_b200.adjoint import DifferentiablePoisson
        problem = DifferentiablePoisson(space, dim, order, cells)
        target = b.roll(1) * math.prod(0.5 / c for c in cells)
        return dict(state, problem=problem, kappas=kappas, b=b, target=target)

    if call in ("embedded", "two_level"):
        mesh = StructuredMesh(dim, order, cells)
        matrix, boundary, dofmap = _pattern(space, mesh)
        assembler = Assembler(space, matrix, mesh, d_dofmap=dofmap)
        # the sphere's centre is what a user moves from call to call
        centre = _centre(case, seed)
        if call == "embedded":
            values = (matrix.entries if case["dtype"] == "f64" else
                      torch.zeros(matrix.nnz(), dtype=torch.float32, device=space.device))
            return dict(state, assembler=assembler, boundary=boundary, centre=centre, b=b, values=values,
                        dtype=case["dtype"], matrix=matrix)
        from cie_b200.twolevel import make_two_level_cg
        assembler.assemble_embedded(centre, RADIUS, ALPHA, DEPTH)
        assembler.dirichlet(boundary, b)
        problem = PoissonProblem(space, mesh, matrix, b, None, boundary, assembler, seed)
        solver = make_two_level_cg(space, problem, _tight(), center=centre, radius=RADIUS, alpha=ALPHA, depth=DEPTH,
                                   degree=6, coarseIterations=80, precision="f32")
        return dict(state, solver=solver, b=b, problem=problem)

    if call == "assemble":
        mesh = StructuredMesh(dim, order, cells)
        matrix, boundary, dofmap = _pattern(space, mesh)
        assembler = Assembler(space, matrix, mesh, d_dofmap=dofmap)
        return dict(state, assembler=assembler, boundary=boundary, kappa=kappas[0], b=b, matrix=matrix)

    if call == "multi":
        matrix, boundary = _system(space, dim, order, cells, kappas[0])[1:3]
        b = torch.where(boundary.bool()[:, None], 0.0, b)  # the load cases as the elimination leaves them
        A = CSROperator(matrix, space)
        solver = MultiRHSConjugateGradients(A, makeDiagonalOperator(matrix, space, csr_handle=A.csr), case["columns"],
                                            _tight())
        if case["dtype"] == "f32":
            solver.set_refinement(0.1)
        return dict(state, solver=solver, b=b)

    matrix = _system(space, dim, order, cells, kappas[0], b)[1]
    if call == "product":
        x = b
        if case["dtype"] == "f32":
            torch.cuda.synchronize()
            space = CUDASpace(torch.float32)
            matrix, x = matrix.astype(torch.float32), x.to(torch.float32)
        return dict(state, space=space, operator=CSROperator(matrix, space), x=x, y=torch.empty_like(x))
    A = CSROperator(matrix, space)
    D = makeDiagonalOperator(matrix, space, csr_handle=A.csr)
    if call == "cg":
        solver = ConjugateGradients(A, space, D, _tight())
    else:
        solver = MixedPrecisionCG(A, D, _tight(), fuseDirection=True)
    return dict(state, solver=solver, b=b)


def run(state):
    call = state["call"]
    if call == "product":
        state["operator"].product(0.0, state["x"], 1.0, state["y"])
        return state["y"]
    if call in ("cg", "mixed", "batch", "multi", "two_level"):
        x = torch.zeros_like(state["b"])
        state["solver"].product(0.0, state["b"], 1.0, x)
        return x
    if call == "assemble":
        b = state["b"].clone()
        state["assembler"].assemble(state["kappa"])
        state["assembler"].dirichlet(state["boundary"], b)
        return {"entries": state["matrix"].entries, "b": b}
    if call == "embedded":
        assembler, values = state["assembler"], state["values"]
        if state["dtype"] == "f64":
            b = state["b"].clone()
            assembler.assemble_embedded(state["centre"], RADIUS, ALPHA, DEPTH, entries=values)
            assembler.dirichlet(state["boundary"], b, entries=values)
            return {"entries": values, "b": b}
        assembler.assemble_embedded_f32(values, state["centre"], RADIUS, ALPHA, DEPTH)
        assembler.dirichlet_f32(state["boundary"], values)
        return {"entries": values}
    out = []
    for kappa in state["kappas"]:
        kappa = kappa.detach().requires_grad_(True)
        b = state["b"].detach().requires_grad_(True)
        u = state["problem"](kappa, b)
        loss = 0.5 * torch.sum((u - state["target"]) ** 2)
        dk, db = torch.autograd.grad(loss, (kappa, b))
        out.append({"u": u.detach(), "dk": dk, "db": db})
    return out


# ---- what the calls cannot do without ----------------------------------------------------------------

def _entries(dim, order, cells):
    """Rows and stored entries of a structured Q_order matrix."""
    rows = nnz = 1
    for c in cells:
        rows *= order * c + 1
        # vertices couple with two cells (one at the ends), inner nodes with their own
        nnz *= (c - 1) * (2 * order + 1) + 2 * (order + 1) + c * (order - 1) * (order + 1)
    return rows, nnz


def work(case):
    """Inputs read once, outputs written once; the operations of a solve are its iterations' (their number from
    the mesh size, as the condition number of a second-order operator gives it)."""
    call = case["call"]
    if call == "batch":
        bytes_ = flops = 0
        for n in _sizes(case):
            rows, nnz = _entries(2, 2, [n, n])
            bytes_ += 12 * nnz + 4 * rows + 24 * rows
            flops += 8 * n * (2 * nnz + 12 * rows)
        return {"bytes": bytes_, "flops": flops}
    dim, order, cells = case["dim"], case["order"], _cells(case)
    rows, nnz = _entries(dim, order, cells)
    ncells, nb = math.prod(cells), (order + 1) ** dim
    iterations = 3 * order * max(cells)
    step = 2 * nnz + 12 * rows
    if call == "product":
        w = 8 if case["dtype"] == "f64" else 4
        return {"bytes": (w + 4) * nnz + 4 * (rows + 1) + 2 * w * rows, "flops": 2 * nnz}
    if call in ("cg", "mixed"):
        return {"bytes": 12 * nnz + 4 * (rows + 1) + 24 * rows, "flops": iterations * step}
    if call == "multi":
        k = case["columns"]
        return {"bytes": 12 * nnz + 4 * (rows + 1) + (16 * k + 8) * rows, "flops": k * iterations * step}
    if call == "assemble":
        # the element matrices are one reference matrix times a coefficient
        return {"bytes": 8 * nnz + 8 * ncells + 17 * rows + 4 * nb * ncells, "flops": 2 * nb * nb * ncells}
    if call == "embedded":
        w = 8 if case["dtype"] == "f64" else 4
        surface = 4 * math.pi * RADIUS ** 2 * 1.5 * cells[0] ** 2  # cut cells, about
        points = 64 * (order + 1) ** 3
        return {"bytes": w * nnz + 17 * rows + 4 * nb * ncells,
                "flops": 2 * nb * nb * ncells + surface * points * 3 * nb * nb}
    if call == "adjoint":
        one = 12 * nnz + 4 * (rows + 1) + 40 * rows + 16 * ncells + 4 * nb * ncells
        return {"bytes": 2 * one, "flops": 4 * 1.2 * iterations * step}
    return {"bytes": 18 * nnz + 4 * (rows + 1) + 24 * rows, "flops": 40 * cells[0] * 14 * 2 * nnz}


# ---- the same results in 64 bits, in plain torch -----------------------------------------------------

def _centre(case, seed):
    """The sphere's centre, near the box centre, from the seed."""
    rng = random.Random(seed * 1009 + 5)
    return [0.5 + rng.uniform(-0.02, 0.02) for _ in range(case["dim"])]


def _basis(order, x):
    """Lagrange values and derivatives on equispaced nodes of [-1, 1] at the points x: two (points, nodes) arrays."""
    nodes = np.linspace(-1.0, 1.0, order + 1)
    value, slope = np.zeros((len(x), order + 1)), np.zeros((len(x), order + 1))
    for i in range(order + 1):
        others = [j for j in range(order + 1) if j != i]
        value[:, i] = np.prod([(x - nodes[j]) / (nodes[i] - nodes[j]) for j in others], axis=0)
        for m in others:
            rest = [j for j in others if j != m]
            slope[:, i] += np.prod([(x - nodes[j]) / (nodes[i] - nodes[j]) for j in rest], axis=0) / (nodes[i] - nodes[m])
    return value, slope


def _gradients(dim, order, base=None, length=2.0):
    """Tensor Gauss points of the box base + [0, length]^dim in cell coordinates (points, dim), their weights, and
    the parametric basis gradients (points, nodes, dim); first axis fastest."""
    gx, gw = np.polynomial.legendre.leggauss(order + 1)
    base = [-1.0] * dim if base is None else base
    axes = [base[d] + 0.5 * length * (gx + 1.0) for d in range(dim)]
    tables = [_basis(order, a) for a in axes]
    q = np.stack(np.meshgrid(*[np.arange(order + 1)] * dim, indexing="ij")[::-1], axis=-1).reshape(-1, dim)
    points = np.stack([axes[d][q[:, d]] for d in range(dim)], axis=1)
    weights = np.prod([gw[q[:, d]] for d in range(dim)], axis=0) * (0.5 * length) ** dim
    gradients = np.ones((len(q), len(q), dim))
    for axis in range(dim):
        for d in range(dim):
            table = tables[d][1 if d == axis else 0]
            gradients[:, :, axis] *= table[q[:, d]][:, q[:, d]]
    return points, weights, gradients


def _element(dim, order, cells):
    """The stiffness matrix of a cell with kappa = 1: prod(2/h) sum w G G^T with parametric gradients."""
    _, w, G = _gradients(dim, order)
    K = np.einsum("p,pid,pjd->ij", w, G, G) * math.prod(2.0 * c for c in cells)
    return torch.as_tensor(K, device="cuda")


def _dofs(dim, order, cells):
    """Node numbers of every cell (cells, nodes) and the boundary flags of the nodes; first axis fastest."""
    n = [order * c + 1 for c in cells]
    index = torch.zeros((), dtype=torch.int64, device="cuda")
    local = torch.zeros((), dtype=torch.int64, device="cuda")
    boundary = torch.zeros(tuple(reversed(n)), dtype=torch.bool, device="cuda")
    stride = 1
    for d in range(dim):
        shape = [1] * dim
        shape[dim - 1 - d] = -1
        index = index + (torch.arange(cells[d], device="cuda") * (order * stride)).reshape(shape)
        local = local + (torch.arange(order + 1, device="cuda") * stride).reshape(shape)
        boundary.index_fill_(dim - 1 - d, torch.tensor([0, n[d] - 1], device="cuda"), True)
        stride *= n[d]
    return index.reshape(-1, 1) + local.reshape(1, -1), boundary.reshape(-1)


def _matrix(dofs, boundary, elements):
    """The eliminated CSR matrix of element matrices (cells, nodes, nodes), in 64 bits."""
    n, nb = boundary.numel(), dofs.shape[1]
    key = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    key, at = torch.unique(key, return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda")
    val.index_add_(0, at, elements.reshape(-1))
    row, col = key // n, key % n
    on = boundary[row] | boundary[col]
    val = torch.where(on, (row == col).to(torch.float64), val)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    diagonal = torch.zeros(n, dtype=torch.float64, device="cuda")
    diagonal[row[row == col]] = val[row == col]
    return torch.sparse_csr_tensor(rowptr, col, val, (n, n)), diagonal


def _poisson(dim, order, cells, kappa):
    dofs, boundary = _dofs(dim, order, cells)
    K = _element(dim, order, cells)
    return (*_matrix(dofs, boundary, kappa[:, None, None] * K), boundary)


def _solve(A, diagonal, b, tolerance=1e-15, most=20000):
    """Jacobi-preconditioned conjugate gradients on all columns at once, restarted once from the true residual."""
    flat = b.dim() == 1
    b = b.reshape(b.shape[0], -1)
    inverse = (1.0 / diagonal)[:, None]
    x = torch.zeros_like(b)
    for _ in range(2):
        r = b - A @ x
        z = inverse * r
        p, rz = z.clone(), (r * z).sum(0)
        for k in range(most):
            q = A @ p
            alpha = rz / (p * q).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            z = inverse * r
            new = (r * z).sum(0)
            if k % 16 == 15 and bool(((r * r).sum(0).sqrt() <= tolerance * (b * b).sum(0).sqrt()).all()):
                break
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
    return x.reshape(-1) if flat else x


def _inside(points, cells, centre):
    """Whether each of (points, dim) cell coordinates lies in the sphere, for every cell: (cells, points)."""
    dim = len(cells)
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for d in range(dim):
        shape = [1] * dim + [-1]
        shape[dim - 1 - d] = cells[d]
        x = (torch.arange(cells[d], device="cuda", dtype=torch.float64)[:, None] +
             0.5 * (torch.as_tensor(points[:, d], device="cuda")[None, :] + 1.0)) / cells[d]
        total = total + ((x - centre[d]) ** 2).reshape(shape)
    return (total < RADIUS ** 2).reshape(-1, points.shape[0])


def _finite_cells(dim, order, cells, centre):
    """Element matrices of the finite-cell sphere: whole cells by the Gauss rule of the cell, cut cells on the tree
    that halves every box whose points lie on both sides, to DEPTH; a box below the cell that lies outside adds
    nothing unless it is a leaf of the last level."""
    nb = (order + 1) ** dim
    scale = math.prod(2.0 * c for c in cells)
    pts, _, _ = _gradients(dim, order)
    side = _inside(pts, cells, centre)
    whole, none = side.all(1), ~side.any(1)
    K = _element(dim, order, cells)
    elements = torch.where(whole, 1.0, ALPHA).to(torch.float64)[:, None, None] * K
    at = torch.nonzero(~whole & ~none).reshape(-1)
    cut = torch.zeros((at.numel(), nb * nb), dtype=torch.float64, device="cuda")

    def visit(base, length, depth, live):
        p, w, G = _gradients(dim, order, base, length)
        G = torch.as_tensor(np.einsum("p,pid,pjd->pij", w, G, G).reshape(len(w), -1) * scale, device="cuda")
        s = _inside(p, cells, centre)[at]
        same_in, same_out = s.all(1), ~s.any(1)
        last = depth == DEPTH
        keep = live & (same_in | last)
        weight = torch.where(s, 1.0, ALPHA).to(torch.float64) * keep[:, None]
        cut.add_(weight @ G)
        if last:
            return
        live = live & ~same_in & ~same_out
        for child in range(1 << dim):
            visit([base[d] + ((child >> d) & 1) * 0.5 * length for d in range(dim)], 0.5 * length, depth + 1, live)

    every = torch.ones(at.numel(), dtype=torch.bool, device="cuda")
    for child in range(1 << dim):
        visit([-1.0 + ((child >> d) & 1) for d in range(dim)], 1.0, 1, every)
    elements[at] = cut.reshape(-1, nb, nb)
    return elements


def exact(case, seed):
    call = case["call"]
    if call == "batch":
        out = []
        for n, (kappa, b) in zip(_sizes(case), _inputs(case, seed)):
            A, diagonal, boundary = _poisson(2, 2, [n, n], kappa)
            out.append(_solve(A, diagonal, torch.where(boundary, 0.0, b)))
        return torch.cat(out)
    dim, order, cells = case["dim"], case["order"], _cells(case)
    kappas, b = _inputs(case, seed)
    if call in ("embedded", "two_level"):
        dofs, boundary = _dofs(dim, order, cells)
        A, diagonal = _matrix(dofs, boundary, _finite_cells(dim, order, cells, _centre(case, seed)))
        b = torch.where(boundary, 0.0, b)
        if call == "two_level":
            return _solve(A, diagonal, b)
        return {"entries": A.values(), "b": b} if case["dtype"] == "f64" else {"entries": A.values()}
    if call == "adjoint":
        target = b.roll(1) * math.prod(0.5 / c for c in cells)
        dofs, boundary = _dofs(dim, order, cells)
        K = _element(dim, order, cells)
        out = []
        for kappa in kappas:
            A, diagonal = _matrix(dofs, boundary, kappa[:, None, None] * K)
            u = _solve(A, diagonal, torch.where(boundary, 0.0, b))
            lam = _solve(A, diagonal, torch.where(boundary, 0.0, u - target))
            dk = -torch.einsum("ei,ij,ej->e", lam[dofs], K, u[dofs])
            out.append({"u": u, "dk": dk, "db": lam})
        return out
    A, diagonal, boundary = _poisson(dim, order, cells, kappas[0])
    if call == "assemble":
        return {"entries": A.values(), "b": torch.where(boundary, 0.0, b)}
    b = torch.where(boundary if b.dim() == 1 else boundary[:, None], 0.0, b)
    if call == "multi":
        return _solve(A, diagonal, b)
    if call == "product":
        if case["dtype"] == "f32":
            n = A.shape[0]
            A = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values().float().double(), (n, n))
            b = b.float().double()
        return A @ b
    return _solve(A, diagonal, b)
