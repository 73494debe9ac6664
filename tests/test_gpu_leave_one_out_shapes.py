"""`hdfe_leave_one_out` and `hdfe_pair_components` on the shapes their
cooperative passes depend on -- deep trees (one level each barrier), hubs whose
neighbours are dealt over a warp, levels of more vertices than warps, nothing
left alive -- against the oracle (whole numbers, compared exactly)."""

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _path(n):               # worker i joins firms i and i + 1
    w = np.repeat(np.arange(n), 2)
    return w, w + np.tile([0, 1], n)


def _cycle(n):
    w, f = _path(n)
    return w, f % n


def _cycles_joined(n):      # two cycles that share the firms of one worker only
    w, f = _cycle(n)
    return np.concatenate((w, w + n, [2 * n, 2 * n])), np.concatenate((f, f + n, [0, n]))


def _hubs(workers, firms, seed):
    # a worker at every firm, a firm of every worker, the rest at random
    rng = np.random.default_rng(seed)
    w = np.concatenate((np.zeros(firms, int), np.arange(workers),
                        rng.integers(0, workers, workers // 2)))
    f = np.concatenate((np.arange(firms), np.zeros(workers, int),
                        rng.integers(0, firms, workers // 2)))
    return w, f


def _sparse(workers, firms, seed):
    rng = np.random.default_rng(seed)
    w = rng.integers(0, workers, 2 * workers)
    return w, (rng.integers(0, firms, 2 * workers) * rng.random(2 * workers) ** 2).astype(int)


CASES = {
    "path": (_path(700), 1), "cycle": (_cycle(1500), 1), "joined": (_cycles_joined(333), 1),
    "one": ((np.array([0]), np.array([0])), 1), "none": (_path(20), 5),
    "hubs": (_hubs(6000, 1700, 1), 1), "hubs2": (_hubs(6000, 1700, 2), 2),
    "sparse": (_sparse(40_000, 9_000, 3), 1), "dense_firms": (_sparse(60_000, 40, 4), 1),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(name):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200.connected import leave_one_out, pair_components
    (w, f), k = CASES[name]
    order = np.lexsort((f, w))
    a, b = w[order].astype(np.uint32), f[order].astype(np.uint32)
    n0, n1 = int(a.max()) + 1, int(b.max()) + 1
    ta, tb = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
    ref_alive, ref_rows, ref = orc.leave_one_out(a, b, n0, n1, (k, k))
    _, ref_labels, ref_comp = orc.largest_connected(a, b, n0, n1, (k, k))
    for _ in range(2):
        alive, info = leave_one_out(ta, tb, n0, n1, (k, k))
        assert np.array_equal(alive.cpu().numpy(), ref_alive)
        assert info["rows"] == ref_rows
        assert {x: info[x] for x in ref} == ref
        labels, comp, _ = pair_components(ta, tb, n0, n1, (k, k))
        assert np.array_equal(labels.cpu().numpy(), ref_labels)
        assert np.array_equal(comp, ref_comp)
