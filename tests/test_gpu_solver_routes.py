"""Which loop a solve takes, on both sides of each rule of the single launch over sliced
rows, and that the solutions agree: with the graph loop's for the FP64 solver, with each
system solved alone for batches.  Both stop at a relative residual of 1e-10; the matrices'
condition numbers are below 1e3, so solutions agree to 1e-6."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

GRAPH_CSR, SLICED, CSR = 0, 4, 5


def device_matrix(m):
    from cie_b200.linalg import CSRMatrix
    m = sp.csr_matrix(m)
    m.sort_indices()
    return CSRMatrix.from_host(m.shape[1], m.indptr, m.indices, m.data)


def symmetric(pattern, seed):
    """A symmetric positive definite matrix with the entries of `pattern`: negative off the
    diagonal, rows that sum to a hundredth of their diagonal."""
    rng = np.random.default_rng(seed)
    p = sp.triu(pattern, 1, format="coo")
    keep = np.unique(p.row.astype(np.int64) * p.shape[0] + p.col)
    r, c = keep // p.shape[0], keep % p.shape[0]
    upper = sp.coo_matrix((-rng.uniform(0.1, 1.0, len(r)), (r, c)), shape=p.shape).tocsr()
    m = upper + upper.T
    return (m + sp.diags(-1.01 * np.asarray(m.sum(1)).ravel() + 1e-3)).tocsr()


def band(n, half):
    return sp.diags([1.0] * half, range(1, half + 1), shape=(n, n))


def scattered(n, k, seed=0):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), k // 2)
    return sp.coo_matrix((np.ones(len(rows)), (rows, rng.integers(0, n, len(rows)))), shape=(n, n)).tocsr() + sp.coo_matrix(
        (np.ones(len(rows)), (rng.integers(0, n, len(rows)), rows)), shape=(n, n)).tocsr()


def tensor(dim, order, cells):
    n = order * cells + 1
    line = sp.lil_matrix((n, n))
    for e in range(cells):
        line[e * order:e * order + order + 1, e * order:e * order + order + 1] = 1.0
    out = line.tocsr()
    for _ in range(dim - 1):
        out = sp.kron(out, line.tocsr(), format="csr")
    return out


def long_rows(n, length, count=1):
    """About 20 entries a row near the diagonal, and `count` rows of about `length` more, the
    first and the last row among them when there are several."""
    rng = np.random.default_rng(n)
    rows = np.repeat(np.arange(n), 10)
    cols = np.minimum(rows + rng.integers(1, 300, len(rows)), n - 1)
    keep = cols > rows
    rows, cols = [rows[keep]], [cols[keep]]
    for r in np.linspace(0, n - 1, count).astype(int) if count > 1 else [n // 2]:
        first = min(max(0, r - length // 2), n - length)
        rows.append(np.full(length, r))
        cols.append(first + np.arange(length))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    m = sp.coo_matrix((np.ones(len(rows)), (rows, cols)), shape=(n, n)).tocsr()
    return m + m.T


@pytest.mark.parametrize("name,pattern,form", [
    ("short rows", lambda: band(3000, 60), SLICED),
    ("rows of 301 on 1,000", lambda: band(1000, 150), SLICED),  # 16 lanes a row there: the same time
    ("rows of 401 on 1,000", lambda: band(1000, 200), CSR),
    ("rows of 301 on 3,000", lambda: band(3000, 150), SLICED),
    ("rows of 801 on 3,000", lambda: band(3000, 400), CSR),
    ("rows of 601, past shared memory", lambda: band(9000, 300), SLICED),
    ("rows of 801, past shared memory", lambda: band(9000, 400), SLICED),
    ("3D order 3, 2 cells", lambda: tensor(3, 3, 2), CSR),
    ("3D order 3, 5 cells", lambda: tensor(3, 3, 5), SLICED),
    ("3D order 4, 2 cells", lambda: tensor(3, 4, 2), CSR),
    ("3D order 4, 3 cells", lambda: tensor(3, 4, 3), SLICED),  # 8 rows of 729, by warps
    ("rows of 1,201, past shared memory", lambda: band(4000, 600), GRAPH_CSR),
    ("3D order 4, 7 cells", lambda: tensor(3, 4, 7), GRAPH_CSR),
    ("a row of 500 among 12,000", lambda: long_rows(12000, 500), SLICED),
    ("a row of 700 among 900", lambda: long_rows(900, 700), CSR),
    ("a row of 3,000 among 12,000", lambda: long_rows(12000, 3000), SLICED),
    ("8 rows of 800 among 20,001", lambda: long_rows(20001, 800, 8), SLICED),
    ("9 rows of 800 among 20,001", lambda: long_rows(20001, 800, 9), SLICED),  # few lanes a row there
    ("9 rows of 800 among 2,001", lambda: long_rows(2001, 800, 9), CSR),
    ("8 rows of 2,000, past shared memory", lambda: long_rows(140000, 2000, 8), SLICED),
    ("scattered, 4,000 rows of 6", lambda: scattered(4000, 6), SLICED),
    ("scattered, 9,000 rows of 6", lambda: scattered(9000, 6), CSR),
    ("scattered, 9,000 rows of 60", lambda: scattered(9000, 60), SLICED),
])
@pytest.mark.parametrize("preconditioned", [True, False])
def test_single_system(name, pattern, form, preconditioned):
    from cie_b200._lib import call
    from cie_b200.linalg import ConjugateGradients, CSROperator, CUDASpace, Statistics, makeDiagonalOperator
    m = symmetric(pattern(), 3)
    space = CUDASpace()
    matrix = device_matrix(m)
    A = CSROperator(matrix, space)
    D = makeDiagonalOperator(matrix, space, csr_handle=A.csr) if preconditioned else None
    b = torch.as_tensor(np.random.default_rng(5).uniform(-1, 1, m.shape[0])).cuda()
    out = []
    for loop in (0, 1):
        solver = ConjugateGradients(A, space, D, Statistics(5000, 0.0, 1e-10))
        solver.set_loop(loop)
        x = torch.zeros_like(b)
        solver.product(0.0, b, 1.0, x)
        out.append(x.cpu().numpy())
        got = ctypes.c_int()
        call("ciecu_pcg_form", solver._solver, ctypes.byref(got))
        print(name, m.shape[0], m.nnz, np.diff(m.indptr).max(), got.value, solver.getStats().iterationCount)
        assert got.value == (form, GRAPH_CSR)[loop]
        assert np.linalg.norm(m @ out[-1] - b.cpu().numpy()) <= 2e-10 * float(torch.linalg.norm(b))
    assert np.linalg.norm(out[0] - out[1]) <= 1e-6 * np.linalg.norm(out[1])


@pytest.mark.parametrize("order,cells,systems,form", [(1, 8, 592, 1), (1, 8, 593, 0), (1, 16, 1200, 0), (1, 26, 1036, 1),
                                                      (1, 26, 1037, 0), (1, 32, 1100, 1), (1, 2, 5000, 0), (1, 2, 100, 1),
                                                      (12, 2, 5, 1)])
def test_batches(order, cells, systems, form):
    from cie_b200._lib import call
    from cie_b200.linalg import BatchedConjugateGradients, CSRMatrix, CUDASpace, Statistics, makeDiagonalOperator
    m = symmetric(tensor(2, order, cells), 7)
    n, nnz = m.shape[0], m.nnz
    space = CUDASpace()
    s = np.arange(systems, dtype=np.int64)
    scale = 1.0 + 0.001 * (s % 97)
    extents = np.concatenate([(m.indptr[:-1].astype(np.int64)[None] + s[:, None] * nnz).ravel(), [nnz * systems]])
    columns = (m.indices.astype(np.int64)[None] + s[:, None] * n).ravel()
    matrix = CSRMatrix.from_host(n * systems, extents, columns.astype(np.int32), (m.data[None] * scale[:, None]).ravel())
    offsets = np.arange(systems + 1, dtype=np.int64) * n
    b = np.random.default_rng(6).uniform(-1, 1, (systems, n))
    solver = BatchedConjugateGradients(matrix, offsets, space, makeDiagonalOperator(matrix, space),
                                       Statistics(2000, 0.0, 1e-10))
    x = torch.zeros(systems * n, dtype=torch.float64, device="cuda")
    solver.product(0.0, torch.as_tensor(b.ravel()).cuda(), 1.0, x)
    got = ctypes.c_int()
    call("ciecu_batch_form", solver._solver, ctypes.byref(got))
    assert got.value == form
    ref = np.linalg.solve(m.toarray(), b.T).T / scale[:, None]
    err = np.linalg.norm(x.cpu().numpy().reshape(systems, n) - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-6


@pytest.mark.parametrize("counts,form", [((1, 0, 2), 1), ((8, 0, 0), 1),
                                         ((3, 3, 3), 0)])  # too many for warps, and too much padding in slices
def test_batch_with_long_rows(counts, form):
    from cie_b200._lib import call
    from cie_b200.linalg import BatchedConjugateGradients, CUDASpace, Statistics, makeDiagonalOperator
    parts = [symmetric(long_rows(1500 + 130 * k, 700, c) if c else band(900, 12), 11 + k) for k, c in enumerate(counts)]
    space = CUDASpace()
    matrix = device_matrix(sp.block_diag(parts, format="csr"))
    offsets = np.concatenate([[0], np.cumsum([m.shape[0] for m in parts])]).astype(np.int64)
    solver = BatchedConjugateGradients(matrix, offsets, space, makeDiagonalOperator(matrix, space),
                                       Statistics(2000, 0.0, 1e-10))
    b = np.random.default_rng(8).uniform(-1, 1, offsets[-1])
    x = torch.zeros(len(b), dtype=torch.float64, device="cuda")
    solver.product(0.0, torch.as_tensor(b).cuda(), 1.0, x)
    got = ctypes.c_int()
    call("ciecu_batch_form", solver._solver, ctypes.byref(got))
    assert got.value == form
    for k, m in enumerate(parts):
        part = slice(offsets[k], offsets[k + 1])
        ref = np.linalg.solve(m.toarray(), b[part])
        assert np.linalg.norm(x.cpu().numpy()[part] - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("line,plane,n,form", [
    (102, 10302, 1060001, 2), (9, 2707, 1100000, 2), (61, 12205, 1050011, 2), (129, 16641, 1060000, 2),
    (300, 90000, 1080000, 1),   # the halo of a tile costs more than it saves
    (102, 10302, 1040000, 1),   # the upper half fits in L2
])
def test_large_stencils(line, plane, n, form):
    """The graph loop over symmetric 27-diagonal matrices: by marching tiles, or rows of the upper half."""
    from cie_b200._lib import call
    from cie_b200.linalg import ConjugateGradients, CSRMatrix, CSROperator, CUDASpace, Statistics, makeDiagonalOperator
    offsets = torch.tensor(sorted(dz * plane + dy * line + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1)
                                  for dx in (-1, 0, 1)), device="cuda")
    columns = torch.arange(n, device="cuda")[:, None] + offsets
    inside = (columns >= 0) & (columns < n)
    extents = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    extents[1:] = inside.sum(1).cumsum(0).to(torch.int32)
    entries = torch.where(offsets == 0, 28.0, -1.0).to(torch.float64).expand(n, 27)[inside]
    space = CUDASpace()
    matrix = CSRMatrix(n, extents, columns[inside].to(torch.int32), entries)
    A = CSROperator(matrix, space)
    solver = ConjugateGradients(A, space, makeDiagonalOperator(matrix, space, csr_handle=A.csr), Statistics(2, 0.0, 1e-300))
    solver.set_loop(1)
    solver.set_schedule(64)
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    solver.product(0.0, b, 1.0, x)
    got = ctypes.c_int()
    call("ciecu_pcg_form", solver._solver, ctypes.byref(got))
    assert solver.info()["dia_symmetric"] and got.value == form
