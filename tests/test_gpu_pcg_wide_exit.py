"""The wide FP64 PCG's report and solution at every lane width and in both CTA
sizes (512 threads, and 1024 from a million values a vector on): the reported
relative residual is the largest over the columns, computed by the kernel from its
recurrence, within 1e-3 of the host's at a loose tolerance (the recurrence and the
residual part by rounding, 1e-14 of a residual of 1e-6); converged and not; columns
that stop earlier than others; a system cut across warps."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L, k", [(400, 8), (400, 16), (400, 32), (126_000, 5), (126_000, 8),
                                  (63_000, 9), (63_000, 16), (32_000, 17), (32_000, 32)])
def test_report(L, k):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import scipy.sparse as sp
    from hdfe_stream_b200 import gpu
    width = 8 if k <= 8 else 16 if k <= 16 else 32
    assert (L * width >= 1_000_000) == (L > 1000)
    rng = np.random.default_rng(L + k)
    E = 5 * L
    A = sp.coo_matrix((-rng.uniform(0.1, 1.0, E), (rng.integers(0, L, E), rng.integers(0, L, E))),
                      shape=(L, L)).tocsr()
    hub = sp.coo_matrix((np.full(L // 2, -0.01), (np.zeros(L // 2, int),
                                                  rng.integers(0, L, L // 2))), shape=(L, L))
    A = (A + A.T + hub + hub.T).tocsr()                 # row 0: cut across warps
    A = (A + sp.diags(np.abs(A).sum(1).A1 * 1.02 + 1.0)).tocsr()
    A.sort_indices()
    dev = torch.device("cuda", 0)
    b = rng.normal(size=(L, k))
    b[:, k // 2] = A @ np.ones(L)                       # a smooth column
    b[:, 1] = 0.0
    for tol, maxiter in ((1e-6, 500), (1e-30, 3)):
        solver = gpu.BlockSolver(gpu.DeviceCSR.from_scipy(A, dev), 1.0 / A.diagonal(), tol, maxiter)
        for _ in range(5):
            X, its, conv, rel = solver.solve_device(torch.from_numpy(b).to(dev),
                                                    np.arange(k) == 1)
            x = X.cpu().numpy()
            norm = np.linalg.norm(b, axis=0)
            norm[1] = 1.0
            want = (np.linalg.norm(b - A @ x, axis=0) / norm).max()
            assert conv == (tol == 1e-6) and (its == 3) == (tol == 1e-30)
            assert abs(rel - want) <= 1e-3 * want and (rel <= tol) == conv
            assert not x[:, 1].any()
