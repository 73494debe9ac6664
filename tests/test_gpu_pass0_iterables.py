"""Pass 0's id columns as any iterable, read once: the rows of the same list."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pass0_columns_from_a_generator():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200 import pass0
    rng = np.random.default_rng(2)
    N = 700
    t = lambda x: torch.as_tensor(x, device="cuda")
    worker, firm, region = (t(rng.integers(0, n, N)) for n in (90, 11, 4))
    spell, V = t(rng.permutation(N)), t(rng.standard_normal((N, 2)))
    want, levels = pass0.pass0(worker, [firm, region], V, sort_only=[spell])
    got, lev = pass0.pass0(worker, (c for c in (firm, region)), V, sort_only=iter([spell]))
    assert got.n_levels == want.n_levels
    assert all(torch.equal(a, b) for a, b in zip(lev, levels, strict=True))
    for name in ("gcode", "codes", "V"):
        assert torch.equal(getattr(got, name), getattr(want, name))
