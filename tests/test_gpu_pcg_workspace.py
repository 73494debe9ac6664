"""The wide PCG on a workspace of exactly the queried size that starts 8 bytes past
a 16-byte boundary: the same iterations as on an aligned one, the solution equal to
the bit (the sums' order does not depend on the addresses)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5, 8, 13, 16, 20, 32])
def test_shifted_workspace(k):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import scipy.sparse as sp
    from hdfe_stream_b200 import _lib, gpu
    lib, rng = _lib.lib(), np.random.default_rng(k)
    L = 3001
    A = sp.random(L, L, 0.002, random_state=k)
    A = (A + A.T).tocsr()
    A = (A + sp.diags(np.abs(A).sum(1).A1 * 1.1 + 0.1)).tocsr()
    A.sort_indices()
    dev = torch.device("cuda", 0)
    S = gpu.DeviceCSR.from_scipy(A, dev)
    dinv = torch.as_tensor(1.0 / A.diagonal(), device=dev)
    b = torch.as_tensor(rng.standard_normal((L, k)), device=dev)
    size = int(lib.hdfe_pcg_workspace_bytes(L, S.nnz, k))
    out = []
    for shift in (0, 8):
        buf = torch.full((size + 256,), 0x5a, dtype=torch.uint8, device=dev)
        ws = buf.data_ptr() + shift
        X = torch.zeros_like(b)
        info = torch.zeros(3, dtype=torch.float64, device=dev)
        _lib.check(lib.hdfe_pcg_solve(
            S.indptr.data_ptr(), S.indices.data_ptr(), S.data.data_ptr(), L, S.nnz,
            dinv.data_ptr(), b.data_ptr(), k, None, None, 1e-12, 500, X.data_ptr(), ws, size,
            info.data_ptr(), _lib.stream_handle()))
        res = _lib.PcgInfo.from_buffer_copy(info.cpu().numpy().tobytes())
        assert res.status == _lib.HDFE_OK and res.converged
        assert bool((buf[:shift] == 0x5a).all()) and bool((buf[shift + size:] == 0x5a).all())
        out.append((X, int(res.iterations)))
    assert out[0][1] == out[1][1] and torch.equal(out[0][0], out[1][0])
