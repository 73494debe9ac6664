"""Pass 0's short paths against the general ones on the same columns: ids of a
small range by bitmap against numpy's unique, rows from one sorted key against
the chain of sorts -- ragged sizes, orders, strides, types, signs, keys that
just fit 64 bits, ties, and the forms that must take the general path."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda", 0)


@pytest.mark.parametrize("n", [1, 31, 33, 4097, 300_001])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.int16, np.uint8, bool])
def test_factorize_ranges(device, n, dtype):
    import torch
    from hdfe_stream_b200 import pass0
    rng = np.random.default_rng(n)
    limit = pass0.RANGE_PER_ID * n + pass0.RANGE_FREE
    for span in (1, 2, 32, 33, 1000, limit, limit + 1):
        if dtype in (np.int16, np.uint8, bool):
            span = min(span, 2 if dtype is bool else 200)
        lo = 0 if dtype in (np.uint8, bool) else -7 if dtype is np.int16 else -(span // 2)
        ids = lo + rng.integers(0, span, n)
        ids[0] = lo
        ids[-1] = lo + span - 1                         # the range's ends
        ids = ids.astype(dtype)
        codes, levels = pass0.factorize(torch.as_tensor(ids, device=device))
        lev, inv = np.unique(ids, return_inverse=True)
        assert np.array_equal(levels.cpu().numpy(), lev) and codes.dtype == torch.int64
        assert np.array_equal(codes.cpu().numpy(), inv)
    if dtype is np.int64:
        ids = np.array([-2 ** 63, 2 ** 63 - 1, 0] * n, np.int64)[:n]
        codes, levels = pass0.factorize(torch.as_tensor(ids, device=device))
        assert np.array_equal(levels.cpu().numpy()[codes.cpu().numpy()], ids)


@pytest.mark.parametrize("form", ["plain", "weights", "float32", "strided", "ties", "one_row",
                                  "no_columns", "float_ids", "extra", "wide_keys"])
def test_rows_from_one_key(device, form, monkeypatch):
    import torch
    from hdfe_stream_b200 import pass0
    rng = np.random.default_rng(3)
    N = 1 if form == "one_row" else 50_001
    worker = rng.permutation(N * 8)[:N] // (1 if form == "wide_keys" else 6) - 1000
    firm = rng.integers(0, 3000, N) * 5
    year = np.arange(N) % (5 if form == "ties" else 100_003)
    V = rng.standard_normal((N, 0 if form == "no_columns" else 3))
    t = lambda x: torch.as_tensor(x, device=device)
    Vt = t(V)
    if form == "float32":
        Vt = Vt.float()
    if form == "strided":
        Vt = t(np.repeat(V, 2, 1))[:, ::2]
    w = t(rng.uniform(0.5, 2.0, N)) if form in ("weights", "ties") else None
    fes = [t(firm.astype(np.int32)), t(year)]
    if form == "float_ids":
        fes[0] = t(np.round(rng.standard_normal(N), 1))
    if form == "wide_keys":                             # 17 bits x 4 > 64: several keys
        fes += [t(rng.permutation(N)), t(rng.permutation(N))]
    extra = [t(rng.permutation(N))] if form == "extra" else []
    taken = []
    short = pass0._rows_by_one_key
    monkeypatch.setattr(pass0, "_rows_by_one_key",
                        lambda *a: taken.append(short(*a)) or taken[-1])
    rows, levels = pass0.pass0(t(worker), fes, Vt, w, sort_only=extra)
    assert (taken[0] is None) == (form in ("ties", "wide_keys"))
    monkeypatch.setattr(pass0, "_rows_by_one_key", lambda *a: None)
    ref, ref_levels = pass0.pass0(t(worker), fes, Vt, w, sort_only=extra)
    for name in ("gcode", "codes", "V", "w"):
        a, b = getattr(rows, name), getattr(ref, name)
        assert (a is None) == (b is None) and (a is None or (torch.equal(a, b)
                                                            and a.dtype == b.dtype
                                                            and a.is_contiguous()))
    assert rows.n_levels == ref.n_levels
    assert all(torch.equal(a, b) for a, b in zip(levels, ref_levels))


def test_sort_in_place(device):
    """Outputs over the inputs, one pass and several."""
    import torch
    from hdfe_stream_b200 import _lib, pass0
    lib = _lib.lib()
    for bits in (5, 20):
        k = torch.randint(0, 2 ** bits, (10_000,), device=device)
        v = torch.arange(10_000, dtype=torch.int32, device=device)
        want, order = torch.sort(k, stable=True)
        ws, size = pass0._workspace(10_000, device)
        _lib.check(lib.hdfe_sort_pairs(k.data_ptr(), v.data_ptr(), 10_000, bits, k.data_ptr(),
                                       v.data_ptr(), ws.data_ptr(), size, _lib.stream_handle()))
        assert torch.equal(k, want) and torch.equal(v.long(), order)
