"""Solvers of different sizes that run the same kernels with different amounts of shared
memory: one created or used after another, and in threads at the same time, leave each
other's launches alone."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def poisson(dim, order, cells, settings=None, seed=0):
    from cie_b200.fem import make_poisson
    from cie_b200.linalg import CSROperator, CUDASpace, makeDiagonalOperator
    space = CUDASpace()
    problem = make_poisson(space, dim, order, cells, seed=seed)
    A = CSROperator(problem.matrix, space)
    return space, problem, A, makeDiagonalOperator(problem.matrix, space, csr_handle=A.csr)


def residual(A, x, b):
    r = b.clone()
    A.product(1.0, x, -1.0, r)
    torch.cuda.synchronize()
    return float(torch.linalg.norm(r) / torch.linalg.norm(b))


def test_coarse_solves_of_two_sizes():
    from cie_b200.fem import make_embedded_poisson
    from cie_b200.linalg import CUDASpace, Statistics
    from cie_b200.twolevel import make_two_level_cg
    space = CUDASpace()
    solvers, outs = [], []
    for cells in (16, 4):  # 17^3 rows in 7 blocks, then 5^3 rows in one
        problem = make_embedded_poisson(space, 3, 2, [cells] * 3, radius=0.4, alpha=1e-6, depth=1, seed=0)
        solver = make_two_level_cg(space, problem, Statistics(50, 0.0, 1e-3), degree=3, coarseIterations=20,
                                   precision="f32")
        m = (cells + 1) ** 3
        b = torch.as_tensor(np.random.default_rng(cells).uniform(-1, 1, m)).cuda()
        out = torch.zeros_like(b)
        solver.coarse_apply(b, out)
        solvers.append((solver, b))
        outs.append(out.clone())
        assert solver.info()["coarse_cluster_active"]
    for (solver, b), first in zip(solvers, outs):  # the larger one again, after the smaller one's set-up
        out = torch.zeros_like(b)
        solver.coarse_apply(b, out)
        assert torch.equal(out, first)


def test_staged_columns_of_two_sizes():
    from cie_b200.linalg import MultiRHSConjugateGradients, Statistics
    solvers = []
    for cells in ([59, 59, 3], [24, 24, 4]):
        _, problem, A, D = poisson(3, 1, cells)
        solver = MultiRHSConjugateGradients(A, D, 32, Statistics(500, 0.0, 1e-9))
        solver.set_refinement(0.1)
        solver.set_format(1)
        b = problem.rhs[:, None] * torch.arange(1, 33, device="cuda", dtype=torch.float64)
        x = torch.zeros_like(b)
        solver.product(0.0, b.contiguous(), 1.0, x)
        solvers.append((solver, b.contiguous(), x, A))
    for solver, b, x, A in solvers:
        solver.set_format(0)
        solver.set_format(1)  # captured again
        again = torch.zeros_like(x)
        solver.product(0.0, b, 1.0, again)
        assert torch.equal(again, x)
        assert residual(A, again[:, 7].contiguous(), b[:, 7].contiguous()) < 1e-8


@pytest.mark.parametrize("kind", ["diagonals", "sliced", "batch"])
def test_threads_with_solvers_of_two_sizes(kind):
    from cie_b200.linalg import (BatchedConjugateGradients, ConjugateGradients, Statistics, block_diagonal,
                                 makeDiagonalOperator)
    work, errors = [], []
    for t in range(4):
        size = (40, 9)[t % 2]
        if kind == "batch":
            space, problem, A, _ = poisson(2, 2, [size, size])
            matrix, offsets = block_diagonal([problem.matrix] * 3)
            D = makeDiagonalOperator(matrix, space)
            solver = BatchedConjugateGradients(matrix, offsets, space, D, Statistics(40, 0.0, 1e-30))
            b = problem.rhs.repeat(3)
        else:
            space, problem, A, D = poisson(2, 1 if kind == "diagonals" else 3, [size, size])
            solver = ConjugateGradients(A, space, D, Statistics(40, 0.0, 1e-30))
            b = problem.rhs
        x = torch.zeros_like(b)
        solver.product(0.0, b, 1.0, x)
        torch.cuda.synchronize()
        work.append((solver, b, x))
    gate = threading.Barrier(4)

    def run(solver, b, x):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                out = torch.zeros_like(b)
                gate.wait()
                for _ in range(400):
                    out.zero_()
                    solver.product(0.0, b, 1.0, out)
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(out, x):
                        errors.append("other bits")
                        return
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []
