"""The bounded waits of the kernels that read shared memory filled by copies or by other
blocks: a wait made to run out (a copy that is left out, bytes that nobody sends; limits
of a millisecond where they can be set) ends the solve with CIECU_ERR_TIMEOUT, soon, and
the same solver then solves as before, bit for bit."""
import ctypes
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MS = 1_000_000
SECOND = 1.0  # far above the waits of one launch, far below those of a loop that ran on


def timed_out(solve, limit=SECOND):
    from cie_b200._lib import CiecuError
    torch.cuda.synchronize()
    begin = time.perf_counter()
    with pytest.raises(CiecuError) as e:
        solve()
    torch.cuda.synchronize()
    assert e.value.status == 5, e.value
    assert time.perf_counter() - begin < limit


@pytest.mark.parametrize("run", [1, 2, 3])
def test_staged_columns(run):
    from cie_b200._lib import call
    from cie_b200.fem import make_poisson
    from cie_b200.linalg import (CSROperator, CUDASpace, MultiRHSConjugateGradients, Statistics,
                                 makeDiagonalOperator)
    space = CUDASpace()
    problem = make_poisson(space, 3, 1, [24, 24, 4], seed=1)
    A = CSROperator(problem.matrix, space)
    solver = MultiRHSConjugateGradients(A, makeDiagonalOperator(problem.matrix, space, csr_handle=A.csr), 32,
                                        Statistics(500, 0.0, 1e-10))
    solver.set_refinement(0.1)
    solver.set_format(1)
    b = (problem.rhs[:, None] * torch.arange(1, 33, device="cuda", dtype=torch.float64)).contiguous()

    def solve():
        x = torch.zeros_like(b)
        solver.product(0.0, b, 1.0, x)
        return x

    first = solve()
    staged = ctypes.c_int()
    call("ciecu_multi_staged", solver._solver, ctypes.byref(staged))
    assert staged.value == 1
    call("ciecu_multi_debug_wait", solver._solver, MS, run)
    timed_out(solve)
    call("ciecu_multi_debug_wait", solver._solver, 2000 * MS, 0)
    assert torch.equal(solve(), first)


@pytest.mark.parametrize("plane", [1, 2, 9])
def test_marching_tiles(plane):
    from cie_b200._lib import call
    from cie_b200.fem import make_poisson
    from cie_b200.linalg import ConjugateGradients, CSROperator, CUDASpace, Statistics, makeDiagonalOperator
    space = CUDASpace()
    problem = make_poisson(space, 3, 1, [103, 100, 101], seed=1)
    A = CSROperator(problem.matrix, space)
    solver = ConjugateGradients(A, space, makeDiagonalOperator(problem.matrix, space, csr_handle=A.csr),
                                Statistics(12, 0.0, 1e-300))
    solver.set_loop(1)
    solver.set_schedule(64)

    def solve():
        x = torch.zeros_like(problem.rhs)
        solver.product(0.0, problem.rhs, 1.0, x)
        return x

    first = solve()
    form = ctypes.c_int()
    call("ciecu_pcg_form", solver._solver, ctypes.byref(form))
    assert form.value == 2
    solver.debug_exchange(MS, plane)
    for _ in range(2):
        timed_out(solve)
    solver.debug_exchange(2000 * MS, 0)
    assert torch.equal(solve(), first)


@pytest.fixture(scope="module")
def two_level():
    from cie_b200.fem import make_embedded_poisson
    from cie_b200.linalg import CUDASpace, Statistics
    from cie_b200.twolevel import make_two_level_cg
    space = CUDASpace()
    problem = make_embedded_poisson(space, 3, 3, [9, 9, 9], radius=0.4, alpha=1e-6, depth=1, seed=0)
    solver = make_two_level_cg(space, problem, Statistics(30, 0.0, 1e-30), degree=4, coarseIterations=20,
                               precision="f32")
    return solver, problem.rhs


def solved(solver, b):
    x = torch.zeros_like(b)
    solver.product(0.0, b, 1.0, x)
    return x


@pytest.mark.parametrize("what", [1, 2, 3])
def test_coarse_cluster(two_level, what):
    """Waits of about a second, up to one after the other in two blocks: a cycle may wait twice as
    long, and a solve ends after its first cycle or the one after."""
    from cie_b200._lib import call
    solver, b = two_level
    coarse = torch.sin(torch.arange(1000, device="cuda", dtype=torch.float64))

    def apply():
        out = torch.zeros_like(coarse)
        solver.coarse_apply(coarse, out)
        return out

    first, alone = solved(solver, b), apply()
    info = solver.info()
    assert info["coarse_cluster_active"] and info["coarse_cluster_ctas"] > 1
    call("ciecu_mgcg_debug_wait", solver.handle, what)
    timed_out(lambda: solved(solver, b), 12 * SECOND)
    timed_out(apply, 6 * SECOND)
    call("ciecu_mgcg_debug_wait", solver.handle, 0)
    assert torch.equal(apply(), alone)  # before a full solve: the timeout was that call's
    assert torch.equal(solved(solver, b), first)


def test_smoother_window():
    """Each launch of a cycle waits twice, about a second each: one step of a sweep of two, so
    that a cycle has three launches, and at most two cycles."""
    from cie_b200._lib import call
    from cie_b200.fem import make_embedded_poisson
    from cie_b200.linalg import CUDASpace, Statistics
    from cie_b200.twolevel import make_two_level_cg
    space = CUDASpace()
    problem = make_embedded_poisson(space, 3, 3, [12, 12, 12], radius=0.4, alpha=1e-6, depth=1, seed=0)
    solver = make_two_level_cg(space, problem, Statistics(30, 0.0, 1e-30), degree=2, coarseIterations=20,
                               precision="f32")
    first = solved(solver, problem.rhs)
    assert solver.info()["smoother_lanes_per_row"] == 4  # the sliced form
    call("ciecu_mgcg_debug_wait", solver.handle, 4)
    timed_out(lambda: solved(solver, problem.rhs), 30 * SECOND)
    call("ciecu_mgcg_debug_wait", solver.handle, 0)
    assert torch.equal(solved(solver, problem.rhs), first)


@pytest.mark.parametrize("exchange", [1, 2, 7])
@pytest.mark.parametrize("cells,systems", [(6, 200), (60, 5)])  # one block a system and more rounds; several blocks
def test_batch_single_launch(cells, systems, exchange):
    from cie_b200._lib import call
    from cie_b200.fem import make_poisson
    from cie_b200.linalg import (BatchedConjugateGradients, CUDASpace, Statistics, block_diagonal, makeDiagonalOperator)
    space = CUDASpace()
    problem = make_poisson(space, 2, 2, [cells, cells], seed=3)
    matrix, offsets = block_diagonal([problem.matrix] * systems)
    solver = BatchedConjugateGradients(matrix, offsets, space, makeDiagonalOperator(matrix, space),
                                       Statistics(300, 0.0, 1e-9))
    b = problem.rhs.repeat(systems)
    first = solved(solver, b)
    form = ctypes.c_int()
    call("ciecu_batch_form", solver._solver, ctypes.byref(form))
    assert form.value == 1
    call("ciecu_batch_debug_exchange", solver._solver, MS, exchange)
    for _ in range(2):
        timed_out(lambda: solved(solver, b))
    call("ciecu_batch_debug_exchange", solver._solver, 0, 0)
    assert torch.equal(solved(solver, b), first)
