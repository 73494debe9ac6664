"""The coefficient-space passes on wide blocks (windows of whole groups, sums
per run) against the same vectors in narrow blocks (a thread to a group):
group sizes at the window's edges and groups without rows, every lane width,
the covariate counts' variants, weights (some groups without any) and the
collect sink.  Both add the same few thousand terms, of magnitude <= 1e4 with
the covariates, in other orders: 1e-12 of the largest entry."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 0, 1, 65, 16, 16, 0, 0, 8, 24, 2, 100] + [1] * 45 + [3, 5, 0, 9] * 30


@pytest.mark.parametrize("D", [1, 2])
@pytest.mark.parametrize("c, B", [(0, 5), (1, 8), (2, 9), (3, 16), (4, 20), (2, 32), (8, 12)])
@pytest.mark.parametrize("weights, sink", [(False, "omega"), (True, "omega"), (True, None)])
def test_wide_blocks_match_narrow_ones(D, c, B, weights, sink):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib
    device = torch.device("cuda", 0)
    lib, rng = _lib.lib(), np.random.default_rng(c * 100 + B)
    f64 = dict(dtype=torch.float64, device=device)
    starts = torch.as_tensor(np.concatenate(([0], np.cumsum(SIZES))), device=device)
    N, G, nlev = int(starts[-1]), len(SIZES), np.array([700, 7][:D], np.int64)
    codes = rng.integers(0, nlev, (N, D))
    codes[:, 0] = np.repeat(codes[::3, 0], 3)[:N]               # runs of three
    codes = torch.as_tensor(codes.astype(np.int32), device=device)
    X = torch.as_tensor(rng.uniform(0, 40, (N, c)), **f64) if c else None
    w = torch.as_tensor(rng.uniform(0.5, 2.0, N), **f64) if weights else None
    if weights:
        w[5:40] = 0.0                                           # whole groups without weight
    omega = torch.as_tensor(rng.uniform(0, 3, N), **f64) if sink else None
    L = int(nlev.sum())
    U, st = (torch.as_tensor(rng.standard_normal((n, B)), **f64) for n in (L, G))
    C = torch.as_tensor(rng.standard_normal((max(c, 1), B)), **f64)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    p = lambda t: None if t is None else t.data_ptr()
    base = (starts.data_ptr(), G, codes.data_ptr(), D, nlev.ctypes.data, p(w), p(X), c)

    def block(j0, j1):
        k = j1 - j0
        u, s, cj = (t[:, j0:j1].contiguous() for t in (U, st, C))
        acc, ax = torch.zeros((L, k), **f64), torch.zeros((max(c, 1), k), **f64)
        _lib.check(lib.hdfe_rows_reduce(*base, s.data_ptr(), None, k, acc.data_ptr(),
                                        ax.data_ptr(), None, status.data_ptr(),
                                        _lib.stream_handle()))
        rows, groups, gs = (torch.full((n, k), -7.0, **f64) for n in (N, G, G))
        acc2, ax2 = torch.zeros((L, k), **f64), torch.zeros((max(c, 1), k), **f64)
        on = omega is not None
        _lib.check(lib.hdfe_rows_project_coef(
            *base, cj.data_ptr() if c else None, u.data_ptr(), s.data_ptr(), k, rows.data_ptr(),
            groups.data_ptr(), p(omega), acc2.data_ptr() if on else None,
            ax2.data_ptr() if on else None, gs.data_ptr() if on else None, status.data_ptr(),
            _lib.stream_handle()))
        torch.cuda.synchronize()
        return acc, ax[:c], rows, groups, gs, acc2, ax2[:c]
    wide = block(0, B)
    narrow = [torch.cat(t, 1) for t in zip(*(block(j, min(j + 4, B)) for j in range(0, B, 4)))]
    assert int(status.item()) == 0
    for name, a, b in zip(("acc", "acc_x", "rows", "groups", "gsum", "sink", "sink_x"), wide,
                          narrow):
        assert a.numel() == 0 or float((a - b).abs().max()) <= 1e-12 * max(
            float(b.abs().max()), 1.0), name
