"""The first launch of a window pass in a process, at the window sizes just under
48 KB: the kernels' static shared memory counts against the limit too, so these
sizes need the limit raised although the window alone stays below it.  Each
size runs in a process of its own (an earlier launch of the same kernel with a
larger window would have raised the limit) and is compared with the same
vectors in blocks of four, which take the narrow passes: both add the same few
hundred terms of magnitude <= 1e4 in other orders, 1e-12 of the largest entry."""

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (dimensions, covariates, vectors, weights): window bytes a CTA
CASES = [(1, 1, 20, False),     # project with the sink: 48,640
         (2, 1, 32, False),     # project with the sink: 49,152
         (4, 2, 8, True),       # spread: 47,104 to 49,152, as the next three
         (4, 3, 8, False),
         (3, 7, 12, True),
         (4, 8, 12, False)]


def check(D, c, B, weights):
    import torch
    from hdfe_stream_b200 import _lib
    dev = torch.device("cuda", 0)
    lib, rng = _lib.lib(), np.random.default_rng(c * 100 + B)
    f64 = dict(dtype=torch.float64, device=dev)
    sizes = [1, 31, 32, 33, 0, 65, 8, 24] + [3, 5, 9] * 20
    starts = torch.as_tensor(np.concatenate(([0], np.cumsum(sizes))), device=dev)
    N, G, nlev = int(starts[-1]), len(sizes), np.array([70, 7, 5, 3][:D], np.int64)
    codes = torch.as_tensor(rng.integers(0, nlev, (N, D)).astype(np.int32), device=dev)
    X = torch.as_tensor(rng.uniform(0, 40, (N, c)), **f64)
    w = torch.as_tensor(rng.uniform(0.5, 2.0, N), **f64) if weights else None
    omega = torch.as_tensor(rng.uniform(0, 3, N), **f64)
    L = int(nlev.sum())
    U, st = (torch.as_tensor(rng.standard_normal((n, B)), **f64) for n in (L, G))
    C = torch.as_tensor(rng.standard_normal((c, B)), **f64)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    base = (starts.data_ptr(), G, codes.data_ptr(), D, nlev.ctypes.data,
            None if w is None else w.data_ptr(), X.data_ptr(), c)

    def block(j0, j1):
        k = j1 - j0
        u, s, cj = (t[:, j0:j1].contiguous() for t in (U, st, C))
        acc, ax = torch.zeros((L, k), **f64), torch.zeros((c, k), **f64)
        _lib.check(lib.hdfe_rows_reduce(*base, s.data_ptr(), None, k, acc.data_ptr(),
                                        ax.data_ptr(), None, status.data_ptr(),
                                        _lib.stream_handle()))
        groups, gs = torch.zeros((G, k), **f64), torch.zeros((G, k), **f64)
        acc2, ax2 = torch.zeros((L, k), **f64), torch.zeros((c, k), **f64)
        _lib.check(lib.hdfe_rows_project_coef(
            *base, cj.data_ptr(), u.data_ptr(), s.data_ptr(), k, None, groups.data_ptr(),
            omega.data_ptr(), acc2.data_ptr(), ax2.data_ptr(), gs.data_ptr(), status.data_ptr(),
            _lib.stream_handle()))
        torch.cuda.synchronize()
        return acc, ax, groups, gs, acc2, ax2
    wide = block(0, B)
    narrow = [torch.cat(t, 1) for t in zip(*(block(j, min(j + 4, B)) for j in range(0, B, 4)))]
    assert int(status.item()) == 0
    for a, b in zip(wide, narrow):
        assert float((a - b).abs().max()) <= 1e-12 * max(float(b.abs().max()), 1.0)


@pytest.mark.parametrize("D, c, B, weights", CASES)
def test_first_launch_of_a_window(D, c, B, weights):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    run = subprocess.run([sys.executable, __file__, str(D), str(c), str(B), str(int(weights))],
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


if __name__ == "__main__":
    sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
    check(*(int(x) for x in sys.argv[1:4]), bool(int(sys.argv[4])))
