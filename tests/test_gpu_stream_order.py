"""Ordering of a space's stream with the caller's: products from several threads on
their own streams, inside a captured graph, and on the space's own stream, each against
the matrix-vector product of the host (whole-number data: exact in FP64 and FP32)."""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def problem(dtype, n=4099, seed=0):
    from cie_b200.linalg import CSRMatrix, CSROperator, CUDASpace
    rng = np.random.default_rng(seed)
    m = sp.diags([rng.integers(1, 9, n - abs(k)) for k in (-3, 0, 5)], (-3, 0, 5), format="csr", dtype=np.float64)
    space = CUDASpace(dtype=dtype)
    dev = [torch.as_tensor(a).cuda() for a in (m.indptr.astype(np.int32), m.indices.astype(np.int32))]
    matrix = CSRMatrix(n, *dev, torch.as_tensor(m.data).to(dtype).cuda())
    return m, CSROperator(matrix, space), rng


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("where", ["threads", "capture", "own stream"])
def test_products_follow_and_precede_the_callers_work(dtype, where):
    m, A, rng = problem(dtype)
    n = m.shape[0]
    xs = rng.integers(-8, 9, (24, n)).astype(np.float64)
    pinned = torch.as_tensor(xs).to(dtype)
    got = np.zeros_like(xs)
    A.product(0.0, pinned[0].cuda(), 1.0, torch.zeros(n, dtype=dtype, device="cuda"))  # chooses its kernel
    torch.cuda.synchronize()

    def run(rows, stream):
        with torch.cuda.stream(stream):
            x = torch.empty(n, dtype=dtype, device="cuda")
            y = torch.zeros(n, dtype=dtype, device="cuda")
            for i in rows:  # one pair of buffers: each step depends on the order both ways
                x.copy_(pinned[i])
                A.product(0.0, x, 1.0, y)
                y.add_(1.0)
                got[i] = y.cpu().numpy()

    if where == "threads":
        threads = [threading.Thread(target=run, args=(range(t, 24, 4), torch.cuda.Stream())) for t in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    elif where == "own stream":
        run(range(24), A.space.stream)
    else:
        x = torch.empty(n, dtype=dtype, device="cuda")
        y = torch.zeros(n, dtype=dtype, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            A.product(0.0, x, 1.0, y)
            y.add_(1.0)
        for i in range(24):
            x.copy_(pinned[i])
            graph.replay()
            got[i] = y.cpu().numpy()
    assert np.array_equal(got, (m @ xs.T).T + 1.0)
