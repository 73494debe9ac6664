"""The null space's blocks are built by the first call and kept: a call on another
stream right behind it, on inputs of its own, finds them complete (the first
stream is held up by a sleep)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_second_stream():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import fit
    from hdfe_stream_b200.leaveout import InverseOperator
    from hdfe_stream_b200.simulate import pass0_layout, simulate_panel
    rows = pass0_layout(simulate_panel(700, 90, 8, spell=(1, 8), p_move=0.01, seed=3))
    drows = fit.DeviceRows.from_rows(rows)
    cells = fit.pass1(drows)
    op = InverseOperator(drows, cells, fit.build_s(cells))
    rng = np.random.default_rng(0)
    lv, st = (torch.as_tensor(rng.standard_normal((n, 4)), device="cuda") for n in (op.L, op.G))
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)                  # about 0.1 s
        first = op.drop_null(lv, st)
    with torch.cuda.stream(b):
        second = op.drop_null(lv, st)
    torch.cuda.synchronize()
    # sums over the blocks in atomic order, entries of order one
    assert all(float((x - y).abs().max()) <= 1e-13 for x, y in zip(first, second))
