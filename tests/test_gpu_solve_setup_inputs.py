"""`solve_setup` on cells of other types, sizes or devices than pass 1's: what the
torch expressions give (core/solve.py:142-146, 294-320), or their refusal -- the
kernel takes addresses and must not see these."""

from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_inputs():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import fit
    rng = np.random.default_rng(0)
    up = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    diag = up(rng.uniform(0.5, 9.0, 100))
    diag[::7] = 0.0
    rhs = up(rng.standard_normal((100, 3)))
    rhs[:, 1] = 1e-14
    ss = up(np.array([4.0, 4.0, 4.0]))
    cells = lambda **kw: SimpleNamespace(**{"diag": diag, "rhs": rhs, "raw_ss": ss, **kw})  # noqa: E731
    dinv, zero = fit.solve_setup(cells())
    assert zero.tolist() == [0, 1, 0]
    for kw in (dict(raw_ss=ss[:1]), dict(raw_ss=ss[0]), dict(raw_ss=ss.float()),
               dict(rhs=rhs.float()), dict(diag=diag.float()), dict(diag=diag.cpu()),
               dict(raw_ss=ss.cpu()[0]), dict(rhs=rhs.T.contiguous().T)):
        d, z = fit.solve_setup(cells(**kw))
        assert z.dtype == torch.uint8 and z.tolist() == [0, 1, 0]
        want = fit.jacobi(kw.get("diag", diag))
        assert d.dtype == want.dtype and torch.equal(d, want)
    for kw in (dict(raw_ss=ss[:2]), dict(raw_ss=ss.cpu())):
        with pytest.raises(RuntimeError):
            fit.solve_setup(cells(**kw))
