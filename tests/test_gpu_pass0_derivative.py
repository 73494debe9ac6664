"""Pass 0 on variables that carry a forward derivative: the derivative's rows are
gathered as the variables' are (the short path takes plain values only)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pass0_forward_derivative():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import torch.autograd.forward_ad as fw
    from hdfe_stream_b200 import pass0
    rng = np.random.default_rng(1)
    N = 500
    t = lambda x: torch.as_tensor(x, device="cuda")
    worker, firm, year = t(rng.integers(0, 60, N)), t(rng.integers(0, 9, N)), t(rng.permutation(N))
    V, dV = t(rng.standard_normal((N, 2))), t(rng.standard_normal((N, 2)))
    with fw.dual_level():
        rows, _ = pass0.pass0(worker, [firm, year], fw.make_dual(V, dV))
        got = fw.unpack_dual(rows.V)
        ref, _ = pass0.pass0(worker, [firm, year], dV)
        assert got.tangent is not None and torch.equal(got.tangent, ref.V)
