"""The row passes of steps 3-4 (`hdfe_resid_moments`, `hdfe_row_effects`,
`hdfe_variance_sums`, `hdfe_row_scores`) at the edges of their windows of 32
rows: groups of 31, 32, 33 and 200 rows, of none and of zero weight, fewer
groups than a warp takes and more than the grid's first deal, against the same
sums in numpy.  Values are of order one and a group has at most 200 rows, so a
sum in any order is good to some 200 * 2^-53 = 2e-14 of its terms; 1e-12 of each
result's norm leaves room for the cancellation in h and e."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy(starts, codes, offs, w, V, gamma, beta, gam_y):
    """With V (m, N): (moments, [resid, alpha, sums], [he, h], variance sums)."""
    G = len(starts) - 1
    grp = np.repeat(np.arange(G), np.diff(starts))

    def mean(x):                    # per row, its group's weighted mean (0 without weight)
        Wg = np.bincount(grp, w, G)
        s = np.bincount(grp, w * x, G)
        return np.divide(s, Wg, out=np.zeros(G), where=Wg > 0)
    R = V - gamma[offs + codes].sum(1).T
    C = R - np.stack([mean(r)[grp] for r in R])
    u = V[0] - beta @ V[1:] - gam_y[offs + codes].sum(1)
    al, y, a = mean(u), V[0], gam_y[offs[0] + codes[:, 0]]
    b = al[grp]
    sums = [np.sum(w * t) for t in (np.ones_like(y), y, a, b, a * a, b * b, a * b)]
    e = C[0] - beta @ C[1:]
    h = C[1:].T
    he = h * (w * e)[:, None]
    sg = np.stack([np.bincount(grp, c, G) for c in he.T])
    iu = np.triu_indices(len(beta))
    var = np.concatenate([M[iu] for M in ((h.T * w) @ h, he.T @ he, sg @ sg.T)]
                         + [[np.sum(w * e * e)]])
    return (C * w) @ C.T, (u - b, al, np.array(sums)), (he, h), var


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("m,D", [(2, 1), (3, 2), (4, 3), (8, 2)])
@pytest.mark.parametrize("sizes", ["edges", "one", "many"])
def test_row_sums(sizes, m, D, weighted):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200 import _lib
    rng = np.random.default_rng(m * 10 + D)
    n = {"edges": np.array([1, 31, 32, 33, 0, 0, 1, 200, 2, 64, 65, 5, 27, 3, 0]),
         "one": np.array([7]),
         "many": rng.integers(1, 12, 60_000)}[sizes]
    starts = np.concatenate(([0], np.cumsum(n))).astype(np.int64)
    G, N = len(n), int(starts[-1])
    nlev = np.array([301, 10, 4][:D], np.int64)
    offs = np.concatenate(([0], np.cumsum(nlev)[:-1]))
    codes = np.stack([rng.integers(0, k, N) for k in nlev], 1)
    V = rng.normal(size=(m, N))
    w = rng.uniform(0.5, 2.0, N) if weighted else np.ones(N)
    if weighted and G > 6:
        w[starts[6]:starts[7]] = 0.0                # a group of zero weight
    gamma = rng.normal(size=(int(nlev.sum()), m))
    beta = rng.normal(size=m - 1)
    gam_y = gamma[:, 0] - gamma[:, 1:] @ beta
    want = _numpy(starts, codes, offs, w, V, gamma, beta, gam_y)

    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    new = lambda *s: torch.full(s, np.nan, dtype=torch.float64, device="cuda")  # noqa: E731
    lib, sh = _lib.lib(), _lib.stream_handle()
    ds, dc, dw, dV = up(starts), up(codes.astype(np.int32)), up(w), up(V)
    dg, db, dgy = up(gamma), up(beta), up(gam_y)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(max(lib.hdfe_assemble_workspace_bytes(m),
                         lib.hdfe_variance_sums_workspace_bytes(m)), dtype=torch.uint8,
                     device="cuda")
    head = (ds.data_ptr(), G, dc.data_ptr(), D, nlev.ctypes.data)
    tail = (dw.data_ptr() if weighted else None, dV.data_ptr(), m, N)
    end = (ws.data_ptr(), ws.numel(), status.data_ptr(), sh)
    k, T = m - 1, (m - 1) * m // 2
    A, resid, alpha, sums = new(m, m), new(N), new(G), new(7)
    he, h, var = new(N, k), new(N, k), new(3 * T + 1)
    _lib.check(lib.hdfe_resid_moments(*head, *tail, dg.data_ptr(), A.data_ptr(), *end))
    _lib.check(lib.hdfe_row_effects(*head, 0, *tail, db.data_ptr(), dgy.data_ptr(),
                                    resid.data_ptr(), alpha.data_ptr(), sums.data_ptr(), *end))
    _lib.check(lib.hdfe_row_scores(*head, *tail, dg.data_ptr(), db.data_ptr(), he.data_ptr(),
                                   h.data_ptr(), status.data_ptr(), sh))
    _lib.check(lib.hdfe_variance_sums(*head, *tail, dg.data_ptr(), db.data_ptr(), var.data_ptr(),
                                      *end))
    assert int(status.item()) == 0
    for got, ref in zip((A, resid, alpha, sums, he, h, var),
                        (want[0], *want[1], *want[2], want[3])):
        got = got.cpu().numpy()
        assert np.isfinite(got).all()
        assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.array_equal(A.cpu().numpy(), A.cpu().numpy().T)
