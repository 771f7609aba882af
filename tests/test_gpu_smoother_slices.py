"""The FP32 smoother's row passes (sliced copy, and the CSR kernels where rows are short):
one iteration of the two-level CG from zero is x = (b, z) / (z, A z) z with z one cycle of
b, formed here in FP64 with scipy.  Row lengths, sizes and bandwidths at the edges of the
copy's slices (8 rows), steps (16 entries), blocks and windows; the smoother matrix changed
between solves; a band too wide for a window.

Bound: a cycle is at most 2 (degree + 1) = 14 passes, each rounding a row of up to 330
entries in 16 chains (21 + 5 additions, 6e-8 each, all terms of a diagonally dominant row
below its diagonal): 14 x 26 x 6e-8 = 2.2e-5 of the largest entry."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BOUND = 2.2e-5


def banded(n, lengths, band, rng):
    """A symmetric, diagonally dominant matrix whose rows hold about `lengths` entries."""
    count = rng.choice(lengths, n) // 2
    rows = np.repeat(np.arange(n), count)
    cols = rows + rng.integers(-band, band + 1, len(rows))
    inside = (cols >= 0) & (cols < n) & (cols != rows)
    rows, cols = rows[inside], cols[inside]
    half = sp.csr_matrix((rng.uniform(-1, 1, len(rows)), (rows, cols)), shape=(n, n))
    m = (half + half.T).tocsr()
    m = (m + sp.diags(np.asarray(abs(m).sum(axis=1)).ravel() + rng.uniform(1, 2, n))).tocsr()
    m.sort_indices()
    return m


def cycle(A, S, dinv, P, dc, lam, degree, ratio, b):
    """z of the two-level cycle: FP64 vectors over the smoother's matrix S."""
    low = lam / ratio
    theta, delta = 0.5 * (lam + low), 0.5 * (lam - low)
    sigma = theta / delta

    def sweep(r):
        rho = 1.0 / sigma
        d = dinv * r / theta
        x = d.copy()
        for _ in range(1, degree):
            new = 1.0 / (2.0 * sigma - rho)
            r = r - S @ d
            d = new * rho * d + 2.0 * new / delta * (dinv * r)
            x = x + d
            rho = new
        return x

    z = sweep(b)
    z = z + P @ ((P.T @ (b - S @ z)) / dc)
    return z + sweep(b - S @ z)


# 4 lanes a row: the sliced copy; 0: whichever CSR kernel is fastest
@pytest.mark.parametrize("n,lengths,band,degree,lanes", [
    (1, [1], 1, 2, 0), (7, [6], 5, 3, 0), (16, [400], 15, 2, 4), (31, [400], 30, 2, 4), (129, [900], 60, 6, 4),
    (1187, [14], 30, 2, 0), (2369, [300], 700, 3, 4), (4097, [200, 260], 4000, 4, 4),
    (20000, [60, 110, 200], 9000, 2, 4), (3001, [5, 9], 40, 3, 0), (60000, [24], 32000, 2, 0),
    (303500, [64], 900, 2, 4)])
def test_one_iteration_is_one_cycle(n, lengths, band, degree, lanes):
    from cie_b200.linalg import CSRMatrix, CSROperator, CUDASpace, Statistics, makeDiagonalOperator
    from cie_b200.twolevel import TwoLevelCG
    rng = np.random.default_rng(n)
    A = banded(n, lengths, band, rng)
    m = (n + 5) // 6
    P = sp.csr_matrix((rng.uniform(0.5, 1.0, n), (np.arange(n), np.arange(n) // 6)), shape=(n, m))
    dc = np.asarray((P.T @ A @ P).diagonal())
    space = CUDASpace()

    def matrix(M, dtype=torch.float64):
        M = M.tocsr()
        M.sort_indices()
        return CSRMatrix(M.shape[1], torch.as_tensor(M.indptr.astype(np.int32)).cuda(),
                         torch.as_tensor(M.indices.astype(np.int32)).cuda(),
                         torch.as_tensor(M.data.copy()).to(dtype).cuda())

    fine, coarse, s32 = matrix(A), matrix(sp.diags(dc)), matrix(A, torch.float32)
    ops = [CSROperator(x, space) for x in (fine, matrix(P), matrix(P.T), coarse)]
    lam, ratio = 2.0, 5.0  # D^-1 A of a diagonally dominant matrix lies in (0, 2)
    solver = TwoLevelCG(ops[0], makeDiagonalOperator(fine, space), ops[1], ops[2], ops[3],
                        makeDiagonalOperator(coarse, space), Statistics(1, 0.0, 1e-300), degree=degree,
                        coarseIterations=1, ratio=ratio, lambdaMax=lam, smoother32=s32)
    dinv = 1.0 / A.diagonal()
    b = rng.uniform(-1, 1, n)
    for scale in (1.0, 1.25):  # the smoother matrix is read anew by every solve
        s32.entries.copy_(torch.as_tensor(A.data * scale).to(torch.float32))
        z = cycle(A, scale * A, dinv, P, dc, lam, degree, ratio, b)
        ref = (b @ z) / (z @ (A @ z)) * z
        x = torch.zeros(n, dtype=torch.float64).cuda()
        solver.product(0.0, torch.as_tensor(b).cuda(), 1.0, x)
        err = np.abs(x.cpu().numpy() - ref).max() / np.abs(ref).max()
        print(n, lengths, scale, "error %.2e" % err, solver.info())
        assert solver.info()["smoother_offsets16"]
        if lanes:
            assert solver.info()["smoother_lanes_per_row"] == lanes
        assert err <= BOUND
