"""The pipelined coarse solve with its products recomputed every 16 iterations, over every
CSR schedule: the iterate after k iterations against Jacobi-PCG in FP64 torch on the same
matrix, at iteration counts around the recomputation.

Bound: 1e-9 of the iterate.  The recurrences of 16 iterations lose some digits of 1e-16 on
a matrix of condition number about 50 (scattered spectrum): far below, and 1e-5 without
the recomputation on the finite-cell matrices that it was made for."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def jacobi_pcg(A, b, iterations):
    d = 1.0 / torch.diagonal(A)
    x, r = torch.zeros_like(b), b.clone()
    u = d * r
    p, rz = u.clone(), r @ u
    for _ in range(iterations):
        q = A @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        u = d * r
        new = r @ u
        p, rz = u + new / rz * p, new
    return x


@pytest.mark.parametrize("schedule", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("iterations", [15, 16, 17, 32, 33])
def test_iterates(schedule, iterations):
    from cie_b200.fem import make_embedded_poisson
    from cie_b200.linalg import CUDASpace, Statistics
    from cie_b200.twolevel import make_two_level_cg
    space = CUDASpace()
    problem = make_embedded_poisson(space, 3, 2, [9, 8, 7], radius=0.4, alpha=1e-3, depth=1, seed=0)
    solver = make_two_level_cg(space, problem, Statistics(5, 0.0, 1e-3), degree=3, coarseIterations=iterations,
                               precision="f32")
    solver.set_coarse_cluster(False)
    coarse = solver._mg.coarseSolver.lhs
    coarse.csr.set_kernel(schedule)
    m = coarse.lhs
    n = m.rowCount()
    A = torch.sparse_csr_tensor(m.rowExtents.long(), m.columnIndices.long(), m.entries, size=(n, n)).to_dense()
    b = torch.as_tensor(np.random.default_rng(iterations).uniform(-1, 1, n)).cuda()
    x = torch.zeros_like(b)
    solver.coarse_apply(b, x)
    assert not solver.info()["coarse_cluster_active"]
    ref = jacobi_pcg(A, b, iterations)
    assert float(torch.linalg.norm(x - ref) / torch.linalg.norm(ref)) <= 1e-9
