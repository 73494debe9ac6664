"""Two copies of the library in one process (a host program's and this package's):
each has kernels of its own, so each raises its own shared-memory limits -- a
window of 53,760 bytes launches in both, with the same sums (1e-12 of the largest:
some ten terms of magnitude <= 100 an entry, in atomic order)."""

import ctypes
import shutil

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_limits_belong_to_the_copy(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib
    rng, B, c = np.random.default_rng(0), 32, 2
    starts = np.arange(0, 401, 8)
    N, G, L = 400, 50, 40
    up = lambda x: torch.as_tensor(x, device="cuda")
    starts, codes = up(starts), up(rng.integers(0, L, (N, 1)).astype(np.int32))
    w, omega, X = up(rng.uniform(0.5, 2, N)), up(rng.uniform(0, 3, N)), up(rng.uniform(0, 4, (N, c)))
    U, C, s = (up(rng.standard_normal((n, B))) for n in (L, c, G))
    nlev, st = np.array([L], np.int64), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = []
    for i in range(2):
        lib = ctypes.CDLL(shutil.copy(_lib.LIB_PATH, tmp_path / f"copy{i}.so"))
        f = lib.hdfe_rows_project_coef
        f.restype, f.argtypes = _lib.SIGNATURES["hdfe_rows_project_coef"]
        groups, gs, acc, ax = (torch.zeros((n, B), dtype=torch.float64, device="cuda")
                               for n in (G, G, L, c))
        assert f(starts.data_ptr(), G, codes.data_ptr(), 1, nlev.ctypes.data, w.data_ptr(),
                 X.data_ptr(), c, C.data_ptr(), U.data_ptr(), s.data_ptr(), B, None,
                 groups.data_ptr(), omega.data_ptr(), acc.data_ptr(), ax.data_ptr(),
                 gs.data_ptr(), st.data_ptr(), _lib.stream_handle()) == _lib.HDFE_OK
        out.append((groups, gs, acc, ax))
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())
