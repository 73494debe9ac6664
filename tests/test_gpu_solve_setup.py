"""The set-up of step 2 (`hdfe_solve_setup`, core/solve.py:142-146, 294-320)
against the same formulas in numpy: the Jacobi weights are one division each,
exactly; the zero flags at a norm of half and twice the bound, where a sum of
squares in any order (relative error under L * 2^-53) decides alike."""

from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,m", [(1, 1), (3, 2), (255, 3), (148 * 256, 1), (148 * 256 + 1, 16),
                                 (100_003, 5)])
def test_setup(L, m):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200 import fit
    rng = np.random.default_rng(L + m)
    diag = rng.uniform(0.5, 9.0, L)
    diag[:: 7] = 0.0
    diag[3:: 11] = 1e-12                # at the bound: no pivot
    diag[5:: 13] = np.nextafter(1e-12, 1.0)
    diag[min(6, L - 1)] = np.nan
    rhs = rng.normal(size=(L, m))
    rhs /= np.linalg.norm(rhs, axis=0)
    raw_ss = rng.uniform(1.0, 4.0, m)
    bound = fit.RHS_ZERO_TOL * np.sqrt(raw_ss)
    side = np.arange(m) % 2
    rhs *= bound * np.where(side, 2.0, 0.5)
    want = side == 0
    if m > 2:                           # nothing, a negative total, no number
        rhs[:, 0] = 0.0
        raw_ss[1] = -1.0
        rhs[0, 2] = np.nan
        want[:3] = [True, False, False]
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    dinv, zero = fit.solve_setup(SimpleNamespace(diag=up(diag), rhs=up(rhs), raw_ss=up(raw_ss)))
    with np.errstate(divide="ignore", invalid="ignore"):
        np.testing.assert_array_equal(dinv.cpu().numpy(), np.where(diag > 1e-12, 1.0 / diag, 0.0))
    np.testing.assert_array_equal(zero.cpu().numpy().astype(bool), want)
