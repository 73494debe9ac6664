"""The null space's removal by blocks (`hdfe_drop_null`) against an orthonormal
basis of the same vectors by QR on the host, on panels of several components
and one, one to three dimensions, one to 40 columns.  A projection of entries
of order one: 1e-13 absolute."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 2, 3])
@pytest.mark.parametrize("p_move, B", [(0.01, 1), (0.01, 40), (0.2, 5), (0.2, 32)])
def test_drop_null_matches_qr(D, p_move, B):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import fit
    from hdfe_stream_b200.leaveout import InverseOperator
    from hdfe_stream_b200.simulate import pass0_layout, simulate_panel
    rows = pass0_layout(simulate_panel(700, 90, 8, spell=(1, 8), p_move=p_move, seed=3),
                        year_fe=D > 1)
    if D == 3:
        extra = np.random.default_rng(1).integers(0, 5, rows.n_rows).astype(np.uint32)
        rows.codes = np.ascontiguousarray(np.column_stack([rows.codes, extra]))
        rows.n_levels = rows.n_levels + [5]
    drows = fit.DeviceRows.from_rows(rows)
    cells = fit.pass1(drows)
    op = InverseOperator(drows, cells, fit.build_s(cells))
    # the reference's vectors, one column each
    root = fit.components(cells, 0)[0].cpu().numpy()
    starts = op.starts.cpu().numpy()[:-1]
    groot = root[rows.codes[starts, 0].astype(np.int64)]
    n, L, cols = rows.n_levels, op.L, []
    for c in np.unique(root):
        v = np.zeros(op.G + L)
        v[:op.G][groot == c] = 1.0
        v[op.G:op.G + n[0]][root == c] = -1.0
        cols.append(v)
    at = op.G + n[0]
    for d in range(1, D):
        v = np.zeros(op.G + L)
        v[op.G:op.G + n[0]] = 1.0
        v[at:at + n[d]] = -1.0
        at += n[d]
        cols.append(v)
    q = np.linalg.qr(np.column_stack(cols))[0]
    rng = np.random.default_rng(5)
    x = rng.standard_normal((op.G + L, B))
    want = x - q @ (q.T @ x)
    lv, st = op.drop_null(torch.as_tensor(x[op.G:], device="cuda"),
                          torch.as_tensor(x[:op.G], device="cuda"))
    got = np.concatenate([st.cpu().numpy(), lv.cpu().numpy()])
    assert np.abs(got - want).max() < 1e-13
    qs, ql = (t.cpu().numpy() for t in op.null_space())
    basis = np.concatenate([qs, ql])
    assert basis.shape == q.shape
    assert np.abs(basis.T @ basis - np.eye(q.shape[1])).max() < 1e-13
    assert np.abs(basis @ (basis.T @ x) - q @ (q.T @ x)).max() < 1e-13
