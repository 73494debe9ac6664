"""`drop_null` and `apply_inverse` on blocks that the kernel must not take by
address -- other types, sizes, vectors, columns to be broadcast, inputs that
record gradients, forward derivatives, vmap --: refused, or the dense basis'
answer (a projection of entries of order one, 1e-12)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def op():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import fit
    from hdfe_stream_b200.leaveout import InverseOperator
    from hdfe_stream_b200.simulate import pass0_layout, simulate_panel
    rows = pass0_layout(simulate_panel(400, 60, 6, spell=(1, 6), p_move=0.02, seed=3))
    drows = fit.DeviceRows.from_rows(rows)
    cells = fit.pass1(drows)
    return InverseOperator(drows, cells, fit.build_s(cells))


def _blocks(op, B, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    return [torch.as_tensor(rng.standard_normal((n, B)), device=op.dev) for n in (op.L, op.G)]


def _project(op, levels, streamed):
    qs, ql = op.null_space()
    o = qs.T @ streamed + ql.T @ levels
    return levels - ql @ o, streamed - qs @ o


def _close(got, want):
    assert all(g.shape == w.shape and float((g - w).abs().max()) <= 1e-12
               for g, w in zip(got, want))


def test_refused(op):
    lv, st = _blocks(op, 3)
    for a, b in ((lv.float(), st), (lv, st.float()), (lv[:-1], st), (lv, st[:-1]),
                 (lv, st[:, :2]), (lv.cpu(), st), (lv, st.cpu())):
        with pytest.raises(RuntimeError):
            op.drop_null(a, b)
    for a, b in ((lv[:-1], st), (lv, st[:-1]), (lv, st[:, :2])):
        with pytest.raises(RuntimeError):
            op.apply_inverse(a, None, b)


def test_other_shapes(op):
    lv, st = _blocks(op, 3)
    _close(op.drop_null(lv, st), _project(op, lv, st))
    _close(op.drop_null(lv[:, 0], st[:, 0]), [t[:, 0] for t in _project(op, lv, st)])
    _close(op.drop_null(lv, st[:, :1]), _project(op, lv, st[:, :1].expand(-1, 3)))
    assert [t.shape[1] for t in op.drop_null(lv[:, :0], st[:, :0])] == [0, 0]
    U, _, U_g, _ = op.apply_inverse(lv, None, st[:, :1])
    U2, _, U_g2, _ = op.apply_inverse(lv, None, st[:, :1].expand(-1, 3))
    assert float((U - U2).abs().max()) <= 1e-8 and float((U_g - U_g2).abs().max()) <= 1e-8


def test_derivatives(op):
    import torch
    import torch.autograd.forward_ad as fw
    lv, st = _blocks(op, 2)
    dl, ds = _blocks(op, 2, 1)
    a, b = lv.clone().requires_grad_(), st.clone().requires_grad_()
    out = op.drop_null(a, b)
    _close(out, _project(op, lv, st))
    torch.autograd.backward(out, (dl, ds))
    _close((a.grad, b.grad), _project(op, dl, ds))          # the projection is symmetric
    with torch.no_grad():
        assert not op.drop_null(a, b)[0].requires_grad
    with fw.dual_level():
        out = op.drop_null(fw.make_dual(lv, dl), fw.make_dual(st, ds))
        _close([fw.unpack_dual(t).tangent for t in out], _project(op, dl, ds))
    out, tangent = torch.func.jvp(op.drop_null, (lv, st), (dl, ds))
    _close(tangent, _project(op, dl, ds))
    many = torch.vmap(op.drop_null)(torch.stack([lv, dl]), torch.stack([st, ds]))
    for i, (x, y) in enumerate(((lv, st), (dl, ds))):
        _close([t[i] for t in many], _project(op, x, y))
