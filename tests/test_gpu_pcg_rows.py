"""The narrow PCG's choice of lanes and nonzeros a lane by the rows' average
length (4 lanes with 6 or 8 in flight, 8 lanes), on both sides of each line, on
one cluster and on the whole GPU, with rows of one nonzero, of exactly a trip and
of one more.  The matrices are diagonally dominant (condition number under 3), so
solves to a relative residual of 1e-12 agree to 3 * 2 * 1e-12 of the solution's
norm; 1e-11 leaves the rounding of the sums."""

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _matrix(L, avg, seed):
    """A symmetric diagonally dominant CSR with about `avg` nonzeros a row."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    E = int(L * (avg - 1) / 2)
    i, j = rng.integers(1, L, E), rng.integers(1, L, E)     # row 0: its diagonal alone
    for r, n in ((1, 23), (2, 24), (3, 31), (4, 32), (5, 33), (6, 64), (7, 300)):
        i = np.concatenate((i, np.full(n, r)))
        j = np.concatenate((j, 10 + rng.choice(L - 10, n, replace=False)))
    A = sp.coo_matrix((-rng.uniform(0.1, 1.0, len(i)), (i, j)), shape=(L, L)).tocsr()
    A = A + A.T
    A.setdiag(0)
    A.eliminate_zeros()
    A = A + sp.diags(2.0 * np.abs(A).sum(1).A1 + 1.0)
    A = A.tocsr()
    A.sort_indices()
    return A


@pytest.mark.parametrize("L", [1500, 21_000])
@pytest.mark.parametrize("avg", [12.0, 17.7, 18.3, 23.7, 24.3, 40.0])
def test_rows_by_average_length(L, avg):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200 import gpu
    A = _matrix(L, avg, int(10 * avg))
    dinv = 1.0 / A.diagonal()
    rng = np.random.default_rng(1)
    S = gpu.DeviceCSR.from_scipy(A, torch.device("cuda", 0))
    for k in (1, 2, 3, 4):
        b = rng.normal(size=(L, k))
        want, _, ok, _ = orc.pcg((A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data),
                                 dinv, b, None, None, 1e-12)
        got, _, conv, rel = gpu.pcg(S, dinv, b, tol=1e-12)
        assert ok and conv and rel <= 1e-12
        assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
