"""The Rademacher row passes (windows of whole groups, signs as bits) against
the explicit-vector passes on the same draws: group sizes at the window's
edges (1, 31, 32, 33, 65 rows and packs that fill 32 exactly), every lane
width, the covariate counts' variants, with and without weights.  Both forms
add the same few thousand terms of magnitude <= 40 in other orders: 1e-12."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 1, 1, 65, 16, 16, 8, 24, 2, 30, 100] + [1] * 45 + [3, 5, 7, 9] * 30


@pytest.fixture(scope="module")
def device():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("D", [1, 2])
@pytest.mark.parametrize("c, B", [(0, 1), (1, 8), (2, 9), (3, 16), (4, 17), (2, 26), (8, 32)])
@pytest.mark.parametrize("weights, root", [(False, 0), (True, 0), (True, 1)])
def test_draws_match_explicit_vectors(device, D, c, B, weights, root):
    import torch
    from hdfe_stream_b200 import _lib
    lib, rng = _lib.lib(), np.random.default_rng(c * 100 + B)
    f64 = dict(dtype=torch.float64, device=device)
    starts = torch.as_tensor(np.concatenate(([0], np.cumsum(SIZES))), device=device)
    N, G, nlev = int(starts[-1]), len(SIZES), np.array([50, 7][:D], np.int64)
    codes = np.stack([np.sort(rng.integers(0, n, N).reshape(-1, 1), 1)[:, 0] // 2 * 2
                      if d == 0 else rng.integers(0, n, N) for d, n in enumerate(nlev)], 1)
    codes[:, 0] = np.repeat(codes[::3, 0], 3)[:N]               # runs of three
    codes = torch.as_tensor(codes.astype(np.int32), device=device)
    X = torch.as_tensor(rng.uniform(0, 40, (N, c)), **f64) if c else None
    w = torch.as_tensor(rng.uniform(0.5, 2.0, N), **f64) if weights else None
    if weights:
        w[5:40] = 0.0                                           # whole groups without weight
    L = int(nlev.sum())
    U = torch.as_tensor(rng.standard_normal((L, B)), **f64)
    C = torch.as_tensor(rng.standard_normal((max(c, 1), B)), **f64)
    seed, first = 12345, 3
    R = torch.empty((N, B), **f64)
    _lib.check(lib.hdfe_rademacher(R.data_ptr(), N, 0, B, seed, first, _lib.stream_handle()))
    p = lambda t: None if t is None else t.data_ptr()
    base = (starts.data_ptr(), G, codes.data_ptr(), D, nlev.ctypes.data, p(w), p(X), c)
    got = []
    for r in (None, R):
        ws = torch.zeros(256, dtype=torch.uint8, device=device)
        acc, ax = torch.empty((L, B), **f64), torch.empty((max(c, 1), B), **f64)
        sq = torch.empty(B, **f64)
        _lib.check(lib.hdfe_rows_center(*base, p(r), B, seed, first, 0, root, acc.data_ptr(),
                                        ax.data_ptr(), sq.data_ptr(), ws.data_ptr(), 256,
                                        _lib.stream_handle()))
        out, mom = torch.empty((N, B), **f64), torch.ones((5, N), **f64)
        _lib.check(lib.hdfe_rows_project(*base, p(C) if c else None, U.data_ptr(), p(r), B, seed,
                                         first, 0, root, N, out.data_ptr(), mom.data_ptr(),
                                         _lib.stream_handle()))
        got.append((acc, ax[:c], sq, out, mom))
    for name, a, b in zip(("acc", "acc_x", "squares", "out", "moments"), *got):
        assert a.numel() == 0 or float((a - b).abs().max()) <= 1e-12 * max(
            float(b.abs().max()), 1.0), name
