"""The FP32 pass over 32 columns that stages operand rows in shared memory, on small
matrices where it runs: three refined iterations against the same in FP64 torch.  Random
entries on every diagonal, across the ends of lines and planes too, so that every staged
row counts; one run of diagonals and three; fewer tiles of 384 rows than SMs and several
for each; last tiles of 1, 53 and 130 rows; both sides of the line length that fits and of
the plane size that splits the runs.

Bound: 2e-5 of each column.  A row sum of 27 terms in FP32 is some 1e-6 of its terms' size
off, three iterations on a matrix of condition number below 3 add little; a wrong entry
or a missing row is 1e-2."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def offsets(line, plane):
    return sorted(dz * plane + dy * line + dx for dz in ((-1, 0, 1) if plane else (0,)) for dy in (-1, 0, 1)
                  for dx in (-1, 0, 1))


@pytest.mark.parametrize("line,plane,n,staged", [
    (25, 625, 3125, 1),          # 9 tiles, the last of 53 rows
    (31, 961, 124930, 1),        # 326 tiles, the last of 130
    (19, 479, 60289, 1),         # a plane that is no multiple of a line, a last tile of 1 row
    (15, 225, 3375, 0),          # one run of all 27: too much for two stages
    (4, 16, 5001, 1),            # ... that fits
    (175, 875, 7893, 1),         # the longest line
    (176, 880, 7893, 0),
    (40, 0, 9001, 1),            # nine diagonals: one run
    (501, 0, 40009, 1),          # ... and three
])
def test_three_iterations(line, plane, n, staged):
    from cie_b200._lib import call
    from cie_b200.linalg import (CSRMatrix, CSROperator, CUDASpace, MultiRHSConjugateGradients, Statistics,
                                 makeDiagonalOperator)
    torch.manual_seed(n)
    offs = offsets(line, plane)
    half = len(offs) // 2
    full = torch.zeros(n, len(offs), dtype=torch.float64, device="cuda")  # entry k of row r: column r + offs[k]
    for k, o in enumerate(offs):
        if o > 0:
            upper = torch.rand(n - o, dtype=torch.float64, device="cuda") - 0.5
            full[:n - o, k] = upper
            full[o:, len(offs) - 1 - k] = upper
    full[:, half] = 2.0 * full.abs().sum(1) + 1.0 + torch.rand(n, dtype=torch.float64, device="cuda")
    columns = torch.arange(n, device="cuda")[:, None] + torch.tensor(offs, device="cuda")
    inside = (columns >= 0) & (columns < n)
    extents = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    extents[1:] = inside.sum(1).cumsum(0).to(torch.int32)
    matrix = CSRMatrix(n, extents, columns[inside].to(torch.int32), full[inside])

    def times(x):
        far = offs[-1]
        padded = torch.zeros(n + 2 * far, 32, dtype=torch.float64, device="cuda")
        padded[far:far + n] = x
        return sum(full[:, k, None] * padded[far + o:far + o + n] for k, o in enumerate(offs))

    space = CUDASpace()
    A = CSROperator(matrix, space)
    solver = MultiRHSConjugateGradients(A, makeDiagonalOperator(matrix, space, csr_handle=A.csr), 32,
                                        Statistics(3, 0.0, 1e-300))
    solver.set_refinement(0.1)
    solver.set_format(1)
    b = torch.rand(n, 32, dtype=torch.float64, device="cuda") - 0.3
    x = torch.zeros_like(b)
    solver.product(0.0, b, 1.0, x)
    assert solver.info()["spmm_format"] == "dia-%d" % len(offs)
    got = ctypes.c_int()
    call("ciecu_multi_staged", solver._solver, ctypes.byref(got))
    assert got.value == staged
    dinv = 1.0 / full[:, half, None]
    ref, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz = z.clone(), (r * z).sum(0)
    for _ in range(3):
        q = times(p)
        alpha = rz / (p * q).sum(0)
        ref += alpha * p
        r -= alpha * q
        z = dinv * r
        new = (r * z).sum(0)
        p, rz = z + new / rz * p, new
    err = torch.linalg.norm(x - ref, dim=0) / torch.linalg.norm(ref, dim=0)
    print(line, plane, n, float(err.max()), solver.refinements()[:2], solver.getStats()[0].iterationCount)
    assert float(err.max()) <= 2e-5
