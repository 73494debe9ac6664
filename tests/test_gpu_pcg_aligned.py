"""The wide PCG's two-columns-a-lane accesses on vectors that start 8 bytes past
a 16-byte boundary, and at odd widths: the same iterations as on aligned ones,
equal to the rounding of one solve (the sums' order does not depend on the
addresses, so 1e-14 of the solution's norm)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5, 7, 8, 15, 16, 31, 32])
@pytest.mark.parametrize("L", [301, 40_000])
def test_unaligned_vectors(L, k):
    torch = pytest.importorskip("torch")
    import scipy.sparse as sp
    from hdfe_stream_b200 import gpu
    rng = np.random.default_rng(k)
    E = 6 * L
    A = sp.coo_matrix((-rng.uniform(0.1, 1.0, E), (rng.integers(0, L, E), rng.integers(0, L, E))),
                      shape=(L, L)).tocsr()
    A = A + A.T
    A = (A + sp.diags(3.0 * np.abs(A).sum(1).A1 + 1.0)).tocsr()
    A.sort_indices()
    dev = torch.device("cuda", 0)
    solver = gpu.BlockSolver(gpu.DeviceCSR.from_scipy(A, dev), 1.0 / A.diagonal(), 1e-12, 500)
    b = torch.from_numpy(rng.normal(size=(L, k))).to(dev)
    x0 = torch.from_numpy(rng.normal(size=(L, k))).to(dev)

    def shifted(t):                         # 8 bytes past the allocation's start
        buf = torch.empty(L * k + 1, dtype=torch.float64, device=dev)
        v = buf[1:].view(L, k)
        v.copy_(t)
        assert v.data_ptr() % 16 == 8
        return v
    for start in (None, x0):
        X = torch.empty_like(b)
        solver.launch(b, None, start, X)
        its = solver.read_info()
        Y = shifted(torch.zeros_like(b))
        solver.launch(shifted(b), None, None if start is None else shifted(start), Y)
        assert solver.read_info() == its and its[1]
        assert float((X - Y).norm()) <= 1e-14 * float(X.norm())
        R = b.cpu().numpy() - A @ X.cpu().numpy()
        assert np.linalg.norm(R) <= 2e-12 * np.linalg.norm(b.cpu().numpy())
