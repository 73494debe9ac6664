"""`hdfe_leave_one_out` on hubs: vertices of so many neighbours that one warp
would hold the grid at a barrier beyond the barrier's limit of a second are
dealt to the whole grid.  Small hubs around the bound (65,536 neighbours) against
the oracle, whole numbers compared exactly; 30M workers of one firm against what
is known by construction."""

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

HUB = 1 << 16


def _two_firms(workers, seed):
    # a firm that everybody works for, others at random, some workers there only
    rng = np.random.default_rng(seed)
    some = rng.random(workers) < 0.9
    w = np.concatenate((np.arange(workers), np.flatnonzero(some)))
    return w, np.concatenate((np.zeros(workers, int), 1 + rng.integers(0, 50, some.sum())))


def _few_firms(workers, firms, seed):
    # every firm a hub
    rng = np.random.default_rng(seed)
    return np.repeat(np.arange(workers), 2), rng.integers(0, firms, 2 * workers)


def _hub_worker(firms, seed):
    # a worker at every firm, the firms in cycles of their own behind it
    rng = np.random.default_rng(seed)
    w = np.concatenate((np.zeros(firms, int), 1 + np.repeat(np.arange(firms), 2)))
    f = np.concatenate((np.arange(firms), rng.integers(0, firms, 2 * firms)))
    return w, f


CASES = {"below": _two_firms(HUB - 1, 1), "at": _two_firms(HUB, 2), "above": _two_firms(HUB + 33, 3),
         "every_firm": _few_firms(300_000, 4, 4), "worker": _hub_worker(HUB + 1000, 5)}


@pytest.mark.parametrize("name", CASES)
def test_hubs_against_oracle(name):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200.connected import leave_one_out
    w, f = CASES[name]
    order = np.lexsort((f, w))
    a, b = w[order].astype(np.uint32), f[order].astype(np.uint32)
    n0, n1 = int(a.max()) + 1, int(b.max()) + 1
    ref_alive, ref_rows, ref = orc.leave_one_out(a, b, n0, n1)
    ta, tb = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
    alive, info = leave_one_out(ta, tb, n0, n1)
    assert np.array_equal(alive.cpu().numpy(), ref_alive)
    assert info["rows"] == ref_rows
    assert {x: info[x] for x in ref} == ref


def test_a_firm_of_thirty_million():
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200.connected import leave_one_out
    n = 30_000_000
    i = torch.arange(n, dtype=torch.int32, device="cuda")
    a = torch.repeat_interleave(i, 2)
    b = torch.stack([torch.zeros_like(i), 1 + i % 3], 1).reshape(-1).contiguous()
    alive, info = leave_one_out(a, b, n, 4)         # three cycles through the first firm
    assert bool(alive.all())
    assert info["rows"] == 2 * n and info["cut"] == 0 and info["rounds"] == 0
