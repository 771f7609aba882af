"""The FP64 CG over symmetric 27-diagonal matrices past L2 (K1 by tiles marching through the
planes, dia_march.cuh): three iterations against the same in FP64 torch.  Random entries on
every diagonal, across the ends of lines and planes too, so that every window entry counts;
row counts that are no multiple of a plane, of a line or of 16 bytes; short, odd and long
lines (the last too long for a tile's halo: dia_rows_sym).

Bound: 1e-12.  Three iterations are a few dozen roundings of 1e-16 per entry, and dot
products of 1e6 terms of one sign whose order differs (1e-16 x 1e3)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("line,plane,n", [(102, 10302, 1060001), (9, 2707, 1100000), (61, 12205, 1050011),
                                          (129, 16641, 1060000), (300, 90000, 1080000)])
def test_three_iterations(line, plane, n):
    from cie_b200.linalg import (ConjugateGradients, CSRMatrix, CSROperator, CUDASpace, Statistics,
                                 makeDiagonalOperator)
    torch.manual_seed(line)
    offsets = sorted(dz * plane + dy * line + dx for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1))
    upper = {o: torch.rand(n, dtype=torch.float64, device="cuda") - 0.5 for o in offsets if o > 0}
    rows = torch.arange(n, device="cuda")
    full = torch.zeros(n, 27, dtype=torch.float64, device="cuda")  # entry k of row r: column r + offsets[k]
    for k, o in enumerate(offsets):
        if o > 0:
            full[:n - o, k] = upper[o][:n - o]
        elif o < 0:
            full[-o:, k] = upper[-o][:n + o]
    full[:, 13] = full.abs().sum(1) + 1.0 + torch.rand(n, dtype=torch.float64, device="cuda")
    cols = rows[:, None] + torch.tensor(offsets, device="cuda")
    inside = (cols >= 0) & (cols < n)
    extents = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    extents[1:] = inside.sum(1).cumsum(0).to(torch.int32)
    matrix = CSRMatrix(n, extents, cols[inside].to(torch.int32), full[inside])

    def times(x):
        padded = torch.zeros(n + 2 * offsets[-1], dtype=torch.float64, device="cuda")
        padded[offsets[-1]:offsets[-1] + n] = x
        y = torch.zeros_like(x)
        for k, o in enumerate(offsets):
            y += full[:, k] * padded[offsets[-1] + o:offsets[-1] + o + n]
        return y

    space = CUDASpace()
    A = CSROperator(matrix, space)
    b = torch.rand(n, dtype=torch.float64, device="cuda") + 0.5
    solver = ConjugateGradients(A, space, makeDiagonalOperator(matrix, space, csr_handle=A.csr), Statistics(3, 0.0, 1e-300))
    solver.set_loop(1)
    solver.set_schedule(64)  # the diagonals
    for scale in (1.0, 2.0):  # the copy follows the matrix
        matrix.entries.copy_(scale * full[inside])
        x = torch.zeros_like(b)
        solver.product(0.0, b, 1.0, x)
        dinv = 1.0 / full[:, 13]  # the diagonal operator's, made before the entries changed
        ref, r = torch.zeros_like(b), b.clone()
        z = dinv * r
        p, rz = z.clone(), r @ z
        for _ in range(3):
            q = scale * times(p)
            alpha = rz / (p @ q)
            ref += alpha * p
            r -= alpha * q
            z = dinv * r
            new = r @ z
            p, rz = z + new / rz * p, new
        err = float(torch.linalg.norm(x - ref) / torch.linalg.norm(ref))
        print(line, plane, n, scale, "%.2e" % err, solver.info())
        assert solver.getStats().iterationCount == 3
        assert err <= 1e-12
