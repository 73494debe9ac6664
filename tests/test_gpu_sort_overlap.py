"""`hdfe_sort_pairs` with outputs that lie over the inputs, crosswise too (the
values' output over the keys, the keys' output over the values): what a stable
sort of copies gives, for no pass, one and several."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 20])
@pytest.mark.parametrize("form", ["vals_over_keys", "keys_over_vals", "shifted"])
def test_outputs_over_inputs(bits, form):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import _lib, pass0
    n = 9001
    gen = torch.Generator("cuda").manual_seed(bits)
    k = torch.randint(0, 2 ** bits, (n,), device="cuda", generator=gen)
    v = torch.randperm(n, device="cuda", generator=gen).to(torch.int32)
    want_k, order = torch.sort(k, stable=True)
    want_v = v[order]
    buf = torch.zeros(4 * n, dtype=torch.int64, device="cuda")      # 8-byte slots
    at = buf.data_ptr()
    keys, vals = at, at + 16 * n
    keys_out, vals_out = {"vals_over_keys": (at + 24 * n, at + 8 * (n // 3)),
                          "keys_over_vals": (at + 16 * n, at + 8 * n),
                          "shifted": (at + 8, at + 24 * n)}[form]
    buf[:n] = k
    buf.view(torch.int32)[4 * n:5 * n] = v
    ws, size = pass0._workspace(n, k.device)
    _lib.check(_lib.lib().hdfe_sort_pairs(keys, vals, n, bits, keys_out, vals_out, ws.data_ptr(),
                                          size, _lib.stream_handle()))
    o = (keys_out - at) // 8
    assert torch.equal(buf[o:o + n], want_k)
    o = (vals_out - at) // 4
    assert torch.equal(buf.view(torch.int32)[o:o + n], want_v)
