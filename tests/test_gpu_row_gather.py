"""The row-gather assembly at the sizes where its paths change: element sizes with
and without a compile-time kernel, more incident cells per row than a group of
lanes holds, rows too long for shared memory, 16-bit positions; the elimination
over column arrays that do not start on a 16-byte boundary; and cut cells
at other orders, rules and depths.  All
against the restatement, with the tolerances of the other assembly tests."""
from types import SimpleNamespace

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests.test_gpu_linalg import dev, host  # noqa: E402


@pytest.fixture(scope="module")
def space():
    from cie_b200.linalg import CUDASpace
    return CUDASpace()


def _assembled(space, mesh, kappa, colors=None):
    from cie_b200.fem import Assembler, csr_pattern
    from cie_b200.linalg import CSRMatrix
    rp, col = csr_pattern(mesh.ncells, mesh.nb, mesh.dofmap, mesh.ndofs)
    m = CSRMatrix(mesh.ndofs, dev(rp, torch.int32), dev(col, torch.int32), dev(np.full(len(col), 7.0)))
    asm = Assembler(space, m, mesh, colors=colors)
    asm.assemble(dev(kappa))
    return rp, col, m, asm


def _reference(restatement, mesh, kappa):
    rp, col = restatement.csr_pattern(mesh.ncells, mesh.nb, mesh.dofmap, mesh.ndofs)
    Ke = np.concatenate([restatement.element_stiffness(mesh.dim, mesh.order, kappa[e], mesh.h)
                         for e in range(mesh.ncells)])
    val, st = restatement.assemble(mesh.ncells, mesh.nb, mesh.dofmap, Ke, rp, col)
    assert st == 0
    return val


@pytest.mark.parametrize("dim,order,cells", [(1, 1, [5]), (1, 4, [3]), (2, 1, [1, 1]), (2, 4, [3, 2]), (3, 1, [1, 1, 1]),
                                             (3, 2, [2, 3, 2]), (3, 4, [2, 1, 2]), (3, 5, [1, 2, 1])])
def test_element_sizes(space, restatement, dim, order, cells):
    from cie_b200.fem import StructuredMesh
    mesh = StructuredMesh(dim, order, cells)
    kappa = np.random.default_rng(order).uniform(0.5, 2.0, mesh.ncells)
    _, _, m, asm = _assembled(space, mesh, kappa)
    ref = _reference(restatement, mesh, kappa)
    assert np.abs(host(m.entries) - ref).max() <= 1e-13 * np.abs(ref).max()
    asm.assemble(dev(kappa), accumulate=True)
    assert np.abs(host(m.entries) - 2 * ref).max() <= 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("cells", [3, 8, 13, 70])
def test_many_cells_at_one_node(space, restatement, cells):
    """A pinwheel of quadrilaterals: node 0 belongs to every cell, so every cell has
    its own colour, row 0 has `cells` incidences and 2 * cells + 1 entries, and one
    node lies in no cell (its row is empty)."""
    ring = np.arange(2 * cells) + 1
    dofmap = np.array([[0, ring[2 * e], ring[(2 * e + 2) % (2 * cells)], ring[2 * e + 1]] for e in range(cells)],
                      dtype=np.int32)
    mesh = SimpleNamespace(dim=2, order=1, ncells=cells, nb=4, dofmap=dofmap.ravel(), ndofs=2 * cells + 2,
                           h=np.array([0.5, 0.25]), cells=np.array([cells, 1], dtype=np.int32))
    kappa = np.random.default_rng(cells).uniform(0.5, 2.0, cells)
    rp, _, m, _ = _assembled(space, mesh, kappa, colors=np.arange(cells))
    assert rp[-1] == rp[-2]
    ref = _reference(restatement, mesh, kappa)
    assert np.abs(host(m.entries) - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("cells", [[1, 1], [6, 5]])
def test_elimination_of_unaligned_columns(space, restatement, cells, offset):
    from cie_b200.fem import Assembler, StructuredMesh, csr_pattern
    from cie_b200.linalg import CSRMatrix
    mesh = StructuredMesh(2, 1, cells)
    rp, col = csr_pattern(mesh.ncells, mesh.nb, mesh.dofmap, mesh.ndofs)
    rng = np.random.default_rng(1)
    val, rhs = rng.uniform(1, 2, len(col)), rng.uniform(1, 2, mesh.ndofs)
    bnd = (rng.uniform(size=mesh.ndofs) < 0.3).astype(np.uint8)
    c = torch.zeros(len(col) + offset, dtype=torch.int32, device="cuda")
    c[offset:] = dev(col, torch.int32)
    m = CSRMatrix(mesh.ndofs, dev(rp, torch.int32), c[offset:], dev(val))
    d_rhs = dev(rhs)
    Assembler(space, m, mesh).dirichlet(torch.as_tensor(bnd).cuda(), d_rhs)
    rows = np.repeat(np.arange(mesh.ndofs), np.diff(rp))
    ref = np.where((bnd[rows] | bnd[col]) != 0, (rows == col).astype(float), val)
    assert np.array_equal(host(m.entries), ref)
    assert np.array_equal(host(d_rhs), np.where(bnd != 0, 0.0, rhs))


@pytest.mark.parametrize("dim,order,cells,depth,quadrature", [(1, 3, [9], 4, 4), (2, 5, [5, 6], 3, 6), (2, 1, [7, 8], 4, 2),
                                                              (3, 2, [5, 4, 5], 1, 5), (3, 1, [6, 6, 6], 3, 2),
                                                              (2, 7, [4, 4], 2, 8)])
def test_cut_cells_of_other_sizes(space, restatement, dim, order, cells, depth, quadrature):
    from cie_b200.fem import Assembler, StructuredMesh, csr_pattern
    from cie_b200.linalg import CSRMatrix
    mesh = StructuredMesh(dim, order, cells)
    rp, col = csr_pattern(mesh.ncells, mesh.nb, mesh.dofmap, mesh.ndofs)
    m = CSRMatrix(mesh.ndofs, dev(rp, torch.int32), dev(col, torch.int32), dev(np.zeros(len(col))))
    asm = Assembler(space, m, mesh, quadratureOrder=quadrature)
    center, radius, alpha = [0.5, 0.47, 0.52][:dim], 0.36, 1e-3
    assert asm.assemble_embedded(center, radius, alpha, depth) > 0
    Ke = []
    for e in range(mesh.ncells):
        at, rest = [], e
        for d in range(dim):
            at.append(rest % cells[d])
            rest //= cells[d]
        pts, w, s = restatement.cut_cell_points(dim, depth, quadrature, center, radius, np.array(at) * mesh.h, mesh.h,
                                                alpha)
        Ke.append(restatement.element_stiffness(dim, order, 1.0, mesh.h, 0, points=pts.ravel(), weights=w * s))
    ref, st = restatement.assemble(mesh.ncells, mesh.nb, mesh.dofmap, np.concatenate(Ke), rp, col)
    assert st == 0
    assert np.allclose(host(m.entries), ref, rtol=1e-12, atol=1e-14 * np.abs(ref).max())
