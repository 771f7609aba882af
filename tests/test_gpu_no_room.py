"""Solves for whose faster form the device has no room: every allocation of a first solve
fails once, in turn; the solve falls back to another form, and so does, or does not, the
next one.  Both reach the tolerance."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["diagonals", "sliced", "batch"])
def test_every_allocation_of_a_solve(kind):
    from cie_b200._lib import call
    from cie_b200.fem import make_poisson
    from cie_b200.linalg import (BatchedConjugateGradients, ConjugateGradients, CSROperator, CUDASpace, Statistics,
                                 block_diagonal, makeDiagonalOperator)
    space = CUDASpace()
    problem = make_poisson(space, 2, 1 if kind == "diagonals" else 3, [14, 11], seed=2)
    A = CSROperator(problem.matrix, space)
    D = makeDiagonalOperator(problem.matrix, space, csr_handle=A.csr)
    settings = Statistics(1000, 0.0, 1e-10)
    b = problem.rhs
    if kind == "batch":
        matrix, offsets = block_diagonal([problem.matrix] * 3)
        A = CSROperator(matrix, space)
        D = makeDiagonalOperator(matrix, space, csr_handle=A.csr)
        b = b.repeat(3)

    def solver():
        if kind == "batch":
            return BatchedConjugateGradients(matrix, offsets, space, D, settings)
        return ConjugateGradients(CSROperator(problem.matrix, space), space, D, settings)

    def reached(s):
        x = torch.zeros_like(b)
        s.product(0.0, b, 1.0, x)
        r = b.clone()
        A.product(1.0, x, -1.0, r)
        torch.cuda.synchronize()
        return float(torch.linalg.norm(r) / torch.linalg.norm(b))

    assert reached(solver()) < 2e-10
    for which in range(1, 21):
        s = solver()
        call("ciecu_debug_fail_allocation", which)
        try:
            assert reached(s) < 2e-10, which
        finally:
            call("ciecu_debug_fail_allocation", 0)
        for _ in range(2):
            assert reached(s) < 2e-10, which
