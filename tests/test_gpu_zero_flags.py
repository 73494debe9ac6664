"""`BlockSolver.launch` and `solve_flagged` by where the zero flags are: host
arrays, lists and CPU tensors as ever, device tensors by `solve_flagged` alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_zero_flags():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import scipy.sparse as sp
    from hdfe_stream_b200 import gpu
    rng = np.random.default_rng(0)
    L, k = 500, 3
    A = sp.random(L, L, 0.01, random_state=1)
    A = (A + A.T + sp.diags(np.full(L, 30.0))).tocsr()
    A.sort_indices()
    dev = torch.device("cuda", 0)
    solver = gpu.BlockSolver(gpu.DeviceCSR.from_scipy(A, dev), 1.0 / A.diagonal(), 1e-12, 500)
    B = torch.as_tensor(rng.standard_normal((L, k)), device=dev)
    flags = np.array([False, True, False])
    out = []
    for zero in (flags, flags.tolist(), torch.as_tensor(flags),
                 torch.as_tensor(flags.astype(np.uint8))):
        X = torch.full_like(B, 7.0)
        solver.launch(B, zero, None, X)
        assert solver.read_info()[1]
        out.append(X)
    out.append(solver.solve_flagged(B, torch.as_tensor(flags.astype(np.uint8), device=dev))[0])
    assert not out[0][:, 1].any() and out[0][:, 0].any()
    assert all(torch.equal(x, out[0]) for x in out[1:])
    with pytest.raises(TypeError):                      # as numpy refuses to read one
        solver.launch(B, torch.as_tensor(flags, device=dev), None, X)
    for bad in (torch.as_tensor(flags), torch.as_tensor(flags, device=dev),
                torch.zeros(2, dtype=torch.uint8, device=dev),
                torch.zeros(6, dtype=torch.uint8, device=dev)[::2]):
        with pytest.raises(ValueError):
            solver.solve_flagged(B, bad)
