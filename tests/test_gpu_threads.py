"""Two host threads, each on a stream of its own, in the same passes on panels
whose windows and tables differ in size: every launch succeeds (a launch must not
depend on a kernel-wide limit that the other thread sets to its own size), and
each thread's sums are what it computes alone, to the rounding of the atomic
order (1e-12 of the largest: some thousand terms of magnitude <= 1e4)."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _panel(torch, dev, nlev, weights, c, B, seed):
    rng = np.random.default_rng(seed)
    f64 = dict(dtype=torch.float64, device=dev)
    sizes = rng.integers(1, 9, 400)
    N, G, D = int(sizes.sum()), len(sizes), len(nlev)
    codes = rng.integers(0, nlev, (N, D))
    order = np.lexsort(tuple(codes.T[::-1]) + (np.repeat(np.arange(G), sizes),))
    p = {"starts": torch.as_tensor(np.concatenate(([0], np.cumsum(sizes))), device=dev),
         "gcode": torch.as_tensor(np.repeat(np.arange(G), sizes).astype(np.int32), device=dev),
         "codes": torch.as_tensor(codes[order].astype(np.int32), device=dev),
         "nlev": np.array(nlev, np.int64), "L": int(sum(nlev)), "N": N, "G": G, "D": D,
         "X": torch.as_tensor(rng.uniform(0, 40, (N, c)), **f64),
         "w": torch.as_tensor(rng.uniform(0.5, 2.0, N), **f64) if weights else None,
         "c": c, "B": B}
    for name, n in (("U", p["L"]), ("s", G), ("C", c)):
        p[name] = torch.as_tensor(rng.standard_normal((n, B)), **f64)
    p["omega"] = torch.as_tensor(rng.uniform(0, 3, N), **f64)
    p["V"] = torch.as_tensor(rng.standard_normal((3, N)), **f64)
    return p


def _passes(torch, lib, _lib, fit, p, sh):
    """One round of the passes on the current stream; their sums."""
    f64 = dict(dtype=torch.float64, device=p["X"].device)
    L, G, N, c, B = p["L"], p["G"], p["N"], p["c"], p["B"]
    base = (p["starts"].data_ptr(), G, p["codes"].data_ptr(), p["D"], p["nlev"].ctypes.data,
            None if p["w"] is None else p["w"].data_ptr(), p["X"].data_ptr(), c)
    status = torch.zeros(1, dtype=torch.int32, device=p["X"].device)
    acc, ax = torch.zeros((L, B), **f64), torch.zeros((c, B), **f64)
    _lib.check(lib.hdfe_rows_reduce(*base, p["s"].data_ptr(), None, B, acc.data_ptr(),
                                    ax.data_ptr(), None, status.data_ptr(), sh))
    acc2, ax2, groups = (torch.zeros((n, B), **f64) for n in (L, c, G))
    _lib.check(lib.hdfe_rows_project_coef(
        *base, p["C"].data_ptr(), p["U"].data_ptr(), p["s"].data_ptr(), B, None,
        groups.data_ptr(), p["omega"].data_ptr(), acc2.data_ptr(), ax2.data_ptr(), None,
        status.data_ptr(), sh))
    k = 8                                           # draws: sixteen windows a CTA
    ws = torch.zeros(256, dtype=torch.uint8, device=p["X"].device)
    acc3, ax3, sq = torch.empty((L, k), **f64), torch.empty((c, k), **f64), torch.empty(k, **f64)
    _lib.check(lib.hdfe_rows_center(*base, None, k, 7, 0, 0, 0, acc3.data_ptr(), ax3.data_ptr(),
                                    sq.data_ptr(), ws.data_ptr(), 256, sh))
    mom = torch.zeros((5, N), **f64)
    u, cj = p["U"][:, :k].contiguous(), p["C"][:, :k].contiguous()
    _lib.check(lib.hdfe_rows_project(*base, cj.data_ptr(), u.data_ptr(), None, k, 7, 0, 0, 0, N,
                                     None, mom.data_ptr(), sh))
    cells = fit.pass1(fit.DeviceRows(p["gcode"], p["codes"], p["V"], p["w"],
                                     [int(n) for n in p["nlev"]]))
    S = fit.build_s(cells)
    assert int(status.item()) == 0
    return [acc, ax, groups, acc2, ax2, acc3, ax3, mom, cells.rhs, S.data]


@pytest.mark.parametrize("first, second", [
    (dict(nlev=[90], weights=False), dict(nlev=[90], weights=True)),
    (dict(nlev=[90, 6], weights=False), dict(nlev=[90, 16], weights=False)),
    (dict(nlev=[90, 6], weights=True), dict(nlev=[90, 6, 5], weights=True))])
def test_two_threads(first, second):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib, fit
    lib, dev = _lib.lib(), torch.device("cuda", 0)
    panels = [_panel(torch, dev, c=2, B=32, seed=i, **kw) for i, kw in enumerate((first, second))]
    alone = [_passes(torch, lib, _lib, fit, p, _lib.stream_handle()) for p in panels]
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(2)

    def run(p, want):
        try:
            stream = torch.cuda.Stream(dev)
            with torch.cuda.stream(stream):
                start.wait(60)
                for _ in range(150):
                    got = _passes(torch, lib, _lib, fit, p, _lib.stream_handle())
                for a, b in zip(got, want):
                    assert a.shape == b.shape
                    assert float((a - b).abs().max()) <= 1e-12 * max(float(b.abs().max()), 1.0)
        except BaseException as e:              # shown by the main thread
            errors.append(e)
    threads = [threading.Thread(target=run, args=(p, a)) for p, a in zip(panels, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors[0]
