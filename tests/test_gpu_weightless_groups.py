"""A group without weight whose streamed value or level's effect is no finite
number: the wide blocks of the coefficient passes (windows, and groups of more
than a window) leave it out of the levels' sums and report a zero group value,
as the narrow blocks do.  Where both are finite, 1e-12 of the largest entry."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [5, 40])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("B", [8, 20])
def test_wide_as_narrow(size, bad, B):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib
    lib, rng = _lib.lib(), np.random.default_rng(B)
    dev = torch.device("cuda", 0)
    f64 = dict(dtype=torch.float64, device=dev)
    sizes = [3, size, 7, 2, size, 4]
    starts = np.concatenate(([0], np.cumsum(sizes)))
    N, G, L, c = int(starts[-1]), len(sizes), 12, 1
    w = rng.uniform(0.5, 2.0, N)
    w[starts[1]:starts[2]] = 0.0                        # the second group
    codes = rng.integers(0, 10, (N, 1))
    codes[starts[1]:starts[2]] = 10 + np.arange(size)[:, None] % 2       # levels of its own
    up = lambda x: torch.as_tensor(x, device=dev)
    starts, codes, w = up(starts), up(codes.astype(np.int32)), up(w)
    X, omega = up(rng.uniform(0, 4, (N, c))), up(rng.uniform(0, 3, N))
    nlev = np.array([L], np.int64)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    base = (starts.data_ptr(), G, codes.data_ptr(), 1, nlev.ctypes.data, w.data_ptr(),
            X.data_ptr(), c)

    def block(U, C, s):
        k = int(s.shape[1])
        acc, ax = torch.zeros((L, k), **f64), torch.zeros((c, k), **f64)
        _lib.check(lib.hdfe_rows_reduce(*base, s.data_ptr(), None, k, acc.data_ptr(),
                                        ax.data_ptr(), None, status.data_ptr(),
                                        _lib.stream_handle()))
        rows, groups, gs = (torch.full((n, k), -7.0, **f64) for n in (N, G, G))
        acc2, ax2 = torch.zeros((L, k), **f64), torch.zeros((c, k), **f64)
        _lib.check(lib.hdfe_rows_project_coef(
            *base, C.data_ptr(), U.data_ptr(), s.data_ptr(), k, rows.data_ptr(),
            groups.data_ptr(), omega.data_ptr(), acc2.data_ptr(), ax2.data_ptr(), gs.data_ptr(),
            status.data_ptr(), _lib.stream_handle()))
        return acc, ax, rows, groups, gs, acc2, ax2
    U, C, s = (up(rng.standard_normal((n, B))) for n in (L, c, G))
    for at in ("streamed", "level"):
        u, st = U.clone(), s.clone()
        if at == "streamed":
            st[1] = bad
        else:
            u[10] = bad
        wide = block(u, C, st)
        narrow = [torch.cat(t, 1) for t in zip(*(block(*(t[:, j:j + 4].contiguous()
                                                         for t in (u, C, st)))
                                                 for j in range(0, B, 4)))]
        assert not wide[3][1].any()
        if at == "streamed":
            assert all(bool(t.isfinite().all()) for t in wide)
        for a, b in zip(wide, narrow):
            fine = b.isfinite()
            assert torch.equal(a.isfinite(), fine)
            if not bool(fine.any()):        # (the covariate block meets every level)
                continue
            assert float((a[fine] - b[fine]).abs().max()) <= 1e-12 * max(
                float(b[fine].abs().max()), 1.0)
