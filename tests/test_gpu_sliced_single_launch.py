"""The single-launch solves over sliced rows (sell_persistent.cuh): FP64 CG on matrices
without a DIA copy, one and several blocks, a last slice of few rows, rows of very
different lengths, odd entry counts, with and without a preconditioner; and batches
whose systems take one block, several, and more rounds than there are blocks.
Diagonally dominant matrices (condition number below 20): the true residual reaches
the 1e-13 that is asked for, and the graph loop's solution agrees to 1e-11."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
sp = pytest.importorskip("scipy.sparse")
pytestmark = pytest.mark.gpu

from tests.test_gpu_linalg import dev, host  # noqa: E402


@pytest.fixture(scope="module")
def space():
    from cie_b200.linalg import CUDASpace
    return CUDASpace()


def random_spd(n, per_row, reach, seed):
    """Random symmetric diagonally dominant matrix, entries within `reach` of the diagonal."""
    rng = np.random.default_rng(seed)
    m = n * per_row // 2
    i = rng.integers(0, n, m)
    j = np.clip(i + rng.integers(-reach, reach + 1, m), 0, n - 1)
    A = sp.coo_matrix((rng.uniform(-1, 1, m), (i, j)), shape=(n, n)).tocsr()
    A = A + A.T
    A = (A + sp.diags([np.asarray(abs(A).sum(axis=1)).ravel() * 1.2 + 1.0], [0])).tocsr()
    A.sum_duplicates()
    A.sort_indices()
    return A


def device(A):
    from cie_b200.linalg import CSRMatrix
    return CSRMatrix(A.shape[1], dev(A.indptr, torch.int32), dev(A.indices, torch.int32), dev(A.data))


CASES = [(40, 30, 39), (128, 20, 60), (129, 9, 100), (1000, 44, 400), (5001, 13, 3000), (60000, 40, 6000),
         (148 * 512 + 1, 50, 9000), (300000, 45, 4000)]


@pytest.mark.parametrize("n,per_row,reach", CASES)
@pytest.mark.parametrize("precond", [True, False])
def test_residual_and_graph_loop(space, n, per_row, reach, precond):
    from cie_b200.linalg import CSROperator, ConjugateGradients, Statistics, makeDiagonalOperator
    A = random_spd(n, per_row, reach, n)
    m = device(A)
    op = CSROperator(m, space)
    assert op.csr.diagonals() == 0
    P = makeDiagonalOperator(m, space, csr_handle=op.csr) if precond else None
    rng = np.random.default_rng(n + 1)
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    solver = ConjugateGradients(op, space, P, Statistics(600, 0.0, 1e-13))
    x = dev(x0)
    solver.product(0.0, dev(b), 2.0, x)
    assert solver.info()["loop"] == "single launch"
    got = host(x) / 2.0
    assert np.linalg.norm(b - A @ got) <= 2e-13 * np.linalg.norm(b - A @ x0)
    graph = ConjugateGradients(op, space, P, Statistics(600, 0.0, 1e-13))
    graph.set_loop(1)
    y = dev(x0)
    graph.product(0.0, dev(b), 2.0, y)
    assert abs(graph.getStats().iterationCount - solver.getStats().iterationCount) <= 2
    assert np.linalg.norm(host(y) / 2.0 - got) <= 1e-11 * np.linalg.norm(got)
    m.entries.mul_(2.0)  # the next solve sees the new values
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    solver2 = solver if P is None else ConjugateGradients(op, space, makeDiagonalOperator(m, space, csr_handle=op.csr),
                                                          Statistics(600, 0.0, 1e-13))
    solver2.product(0.0, dev(b), 1.0, x)
    assert np.linalg.norm(b - 2.0 * (A @ host(x))) <= 2e-13 * np.linalg.norm(b)


def test_wide_matrix_keeps_the_graph(space):
    """A window wider than shared memory does not suit the sliced copy."""
    from cie_b200.linalg import CSROperator, ConjugateGradients, Statistics, makeDiagonalOperator
    A = random_spd(150000, 30, 140000, 3)
    m = device(A)
    op = CSROperator(m, space)
    solver = ConjugateGradients(op, space, makeDiagonalOperator(m, space, csr_handle=op.csr), Statistics(600, 0.0, 1e-13))
    b = np.random.default_rng(1).uniform(-1, 1, 150000)
    x = torch.zeros(150000, dtype=torch.float64, device="cuda")
    solver.product(0.0, dev(b), 1.0, x)
    assert solver.info()["loop"] != "single launch"
    assert np.linalg.norm(b - A @ host(x)) <= 2e-13 * np.linalg.norm(b)


@pytest.mark.parametrize("sizes", [[1], [1, 2, 33], [5000, 200, 31, 32, 33], [70000, 3000, 50000, 1],
                                   [3000] * 200 + [20000] * 40, [17] * 700])
def test_batches(space, sizes):
    from cie_b200.linalg import BatchedConjugateGradients, Statistics, block_diagonal, makeDiagonalOperator
    mats = [random_spd(n, 14, min(500, max(n - 1, 1)), 7 + k) if n > 1 else sp.csr_matrix([[2.5]])
            for k, n in enumerate(sizes)]
    bd, offsets = block_diagonal([device(A) for A in mats])
    rng = np.random.default_rng(len(sizes))
    n = int(offsets[-1])
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    solver = BatchedConjugateGradients(bd, offsets, space, makeDiagonalOperator(bd, space), Statistics(600, 0.0, 1e-13))
    outs = []
    for _ in range(2):
        x = dev(x0)
        solver.product(0.0, dev(b), 1.0, x)
        outs.append(host(x))
    assert np.array_equal(outs[0], outs[1])
    for s, A in enumerate(mats):
        at = slice(int(offsets[s]), int(offsets[s + 1]))
        r0 = np.linalg.norm(b[at] - A @ x0[at])
        assert np.linalg.norm(b[at] - A @ outs[0][at]) <= 2e-13 * r0 + 1e-15, s
