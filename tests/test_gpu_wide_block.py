"""The S build's wide x wide block with more than 16 wide levels: tiles of 32
levels that slide along the wide list (all years of a long panel at once, a
batch's years panel by panel), chunks that meet levels further apart, weights
with a group of none -- against the oracle's S (`_build_explicit`): the same
pattern, values to 1e-12 of the largest (a year's entry sums some 10^4 terms of
one sign: 10^4 * 2^-53 = 1e-12 in the worst order, some 1e-14 in the tiles')."""

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _rows(panels, weights=False, region=0):
    """The panels below one another, levels apart, in pass 0's order."""
    from hdfe_stream_b200.simulate import Rows, pass0_layout
    parts = [pass0_layout(p) for p in panels]
    D = parts[0].codes.shape[1]
    n_levels = [sum(p.n_levels[d] for p in parts) for d in range(D)]
    g0, off, gs, cs = 0, np.zeros(D, np.int64), [], []
    for p in parts:
        gs.append(p.gcode.astype(np.int64) + g0)
        cs.append(p.codes.astype(np.int64) + off)
        g0 += p.n_groups
        off += np.array(p.n_levels[:D])
    g, codes = np.concatenate(gs), np.concatenate(cs)
    V = np.concatenate([p.V for p in parts])
    if region:
        codes = np.column_stack([codes, codes[:, 0] % region])
        n_levels = n_levels + [region]
    w = np.random.default_rng(3).uniform(0.5, 2.0, len(g)) if weights else None
    order = np.lexsort(tuple(V.T[::-1]) + tuple(codes.T[::-1]) + (g,))
    return Rows(gcode=g[order].astype(np.uint32),
                codes=np.ascontiguousarray(codes[order].astype(np.uint32)), V=V[order],
                w=w, n_levels=n_levels, n_groups=g0, names=parts[0].names)


def _panel(workers, T, seed, spell=None):
    from hdfe_stream_b200.simulate import simulate_panel
    return simulate_panel(workers, workers // 20, T, spell=spell or (T // 3, T), p_move=0.2,
                          seed=seed)


@pytest.mark.parametrize("form", ["years17", "years32", "years33", "batch", "uneven", "regions10",
                                  "regions30", "weights"])
def test_many_wide_levels(form):
    pytest.importorskip("torch")
    from hdfe_stream_b200 import fit
    if form.startswith("years"):
        rows = _rows([_panel(20_000, int(form[5:]), 1)])
    elif form == "batch":
        rows = _rows([_panel(6000, 10, s) for s in range(4)])
    elif form == "uneven":              # short spells: chunks meet some of the years only
        rows = _rows([_panel(50_000, 24, 5, spell=(2, 4)), _panel(7000, 12, 6)])
    elif form.startswith("regions"):    # cells with two wide levels, near or far apart
        n = int(form[7:])
        rows = _rows([_panel(2000 * n, 12, 7)], region=n)
    else:
        rows = _rows([_panel(9000, 20, 8), _panel(9000, 9, 9)], weights=True)
    ip, ix, dt = orc.build_explicit(orc.pass1(rows))
    cells = fit.pass1(fit.DeviceRows.from_rows(rows))
    S = fit.build_s(cells)
    assert S.info["n_wide"] > 16
    assert np.array_equal(S.indptr.cpu().numpy(), ip)
    assert np.array_equal(S.indices.cpu().numpy(), ix)
    assert np.max(np.abs(S.data.cpu().numpy() - dt)) <= 1e-12 * np.max(np.abs(dt))
