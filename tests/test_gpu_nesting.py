"""`nested_dims` and `fe_pair_components` against numpy and scipy on coded rows:
nested and loose dimensions, a level without rows, one row off, sizes around
a grid step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 33, 5_000, 700_001])
@pytest.mark.parametrize("off", [False, True])
def test_nesting_and_pair_components(N, off):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    from hdfe_stream_b200 import fit, inference
    rng = np.random.default_rng(N)
    n_cl = max(N // 50, 1)
    firm = rng.integers(0, max(N // 5, 2), N)               # firm f in cluster f % n_cl
    code = firm % n_cl
    if off and N > 1:
        code[N // 2] = (code[N // 2] + 1) % (n_cl + 1)
    other = rng.integers(0, 3, N) + 3 * (firm % 2)          # two blocks of three levels
    used = np.unique(firm)
    firm = np.searchsorted(used, firm)
    nlev = [len(used), 7]                                   # the last of 7 has no rows
    gcode = np.arange(N) // 4
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x.astype(np.int32)), device="cuda")
    rows = fit.DeviceRows(t(gcode), t(np.column_stack([firm, other])),
                          torch.zeros((1, N), dtype=torch.float64, device="cuda"), None, nlev)

    def nested(levels, n):
        lo, hi = np.full(n, 2 ** 60), np.full(n, -1)
        np.minimum.at(lo, levels, code)
        np.maximum.at(hi, levels, code)
        return bool((lo == hi).all())
    got = inference.nested_dims(torch.as_tensor(code, device="cuda"), rows,
                                [int(gcode[-1]) + 1] + nlev)
    assert got == [nested(gcode, gcode[-1] + 1), nested(firm, nlev[0]), nested(other, 7)]
    assert inference.nested_dims(torch.as_tensor(code, device="cuda"), rows,
                                 [None, nlev[0], None]) == [False, nested(firm, nlev[0]), False]
    cells = fit.pass1(rows)
    pair = inference.fe_pair_components(rows, cells)[-1]
    n = sum(nlev)
    want = connected_components(coo_matrix((np.ones(N), (firm, nlev[0] + other)), (n, n)),
                                directed=False)[0]
    assert pair == want
