"""One assembly plan used by several callers at once: threads that assemble with
different conventions, and a captured assembly replayed beside another call.  Every
result is bit for bit the one that a single caller gets."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests.test_gpu_linalg import dev  # noqa: E402


def plan(cells):
    from cie_b200.fem import Assembler, StructuredMesh, csr_pattern
    from cie_b200.linalg import CSRMatrix, CUDASpace
    space = CUDASpace()
    mesh = StructuredMesh(3, 2, cells)
    rp, col = csr_pattern(mesh.ncells, mesh.nb, mesh.dofmap, mesh.ndofs)
    matrix = CSRMatrix(mesh.ndofs, dev(rp, torch.int32), dev(col, torch.int32), dev(np.zeros(len(col))))
    kappa = dev(np.random.default_rng(4).uniform(0.5, 2.0, mesh.ncells))
    assembler = Assembler(space, matrix, mesh)
    alone = []
    for convention in (0, 1):
        out = torch.zeros_like(matrix.entries)
        assembler.assemble(kappa, convention=convention, entries=out)
        alone.append(out)
    torch.cuda.synchronize()
    assert not torch.equal(alone[0], alone[1])
    return assembler, kappa, alone


def test_threads_with_different_conventions():
    assembler, kappa, alone = plan([5, 4, 3])
    wrong = [0, 0, 0, 0]
    gate = threading.Barrier(4)

    def work(t):
        convention = t % 2
        with torch.cuda.stream(torch.cuda.Stream()):
            outs = [torch.zeros_like(alone[0]) for _ in range(8)]
            gate.wait()
            for _ in range(50):
                for out in outs:
                    assembler.assemble(kappa, convention=convention, entries=out)
                torch.cuda.current_stream().synchronize()
                wrong[t] += sum(not torch.equal(out, alone[convention]) for out in outs)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0, 0, 0]


def test_captured_assembly_beside_another_call():
    assembler, kappa, alone = plan([4, 3, 3])
    captured, live = torch.zeros_like(alone[0]), torch.zeros_like(alone[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assembler.assemble(kappa, convention=1, entries=captured)
    other = torch.cuda.Stream()
    for _ in range(200):
        captured.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            graph.replay()
        assembler.assemble(kappa, convention=0, entries=live)
        torch.cuda.synchronize()
        assert torch.equal(captured, alone[1]) and torch.equal(live, alone[0])
