"""Groups without weight whose covariates are no finite numbers, in the centring
pass: the Rademacher form leaves them out of the covariate block as the form of
explicit vectors does (groups inside a window, at its ends and of more than a
window).  The sums of the other groups: some hundred terms of magnitude <= 8,
1e-12 of the largest."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c, B", [(1, 8), (2, 16), (5, 32)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("root", [0, 1])
def test_weightless_groups_add_nothing(c, B, bad, root):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib
    lib, rng = _lib.lib(), np.random.default_rng(B)
    f64 = dict(dtype=torch.float64, device="cuda")
    sizes = [3, 5, 1, 40, 2, 6, 7, 8, 33, 4, 1]
    ends = np.concatenate(([0], np.cumsum(sizes)))
    N, G, nlev = int(ends[-1]), len(sizes), np.array([9, 4], np.int64)
    w, X = rng.uniform(0.5, 2.0, N), rng.uniform(0, 4, (N, c))
    for g in (0, 2, 3, 6, 10):
        w[ends[g]:ends[g + 1]] = 0.0
        X[ends[g]:ends[g + 1]] = bad
    up = lambda x: torch.as_tensor(x, device="cuda")
    starts, w, X = up(ends), up(w), up(X)
    codes = up(np.stack([rng.integers(0, n, N) for n in nlev], 1).astype(np.int32))
    R = torch.empty((N, B), **f64)
    _lib.check(lib.hdfe_rademacher(R.data_ptr(), N, 0, B, 7, 2, _lib.stream_handle()))
    got = []
    for r in (None, R.data_ptr()):
        ws = torch.zeros(256, dtype=torch.uint8, device="cuda")
        acc, ax, sq = (torch.empty((n, B), **f64) for n in (int(nlev.sum()), c, 1))
        _lib.check(lib.hdfe_rows_center(
            starts.data_ptr(), G, codes.data_ptr(), 2, nlev.ctypes.data, w.data_ptr(),
            X.data_ptr(), c, r, B, 7, 2, 0, root, acc.data_ptr(), ax.data_ptr(), sq.data_ptr(),
            ws.data_ptr(), 256, _lib.stream_handle()))
        got.append((acc, ax, sq))
    for a, b in zip(*got):
        assert bool(b.isfinite().all()) and bool(a.isfinite().all())
        assert float((a - b).abs().max()) <= 1e-12 * max(float(b.abs().max()), 1.0)
