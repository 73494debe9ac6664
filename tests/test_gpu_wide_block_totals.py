"""The S build's wide x wide block beyond 16 wide levels where the tiles must not
be used: groups whose total weight is zero, subnormal or so large that its
reciprocal is subnormal, and lists of groups with more groups than cells (empty
ones), which go by atomics alone.  Against the oracle's S (`_build_explicit`) at
the wide levels' entries: no number at the same places, the others to 1e-12 of
the largest finite one (a year's entry sums some 10^4 terms of one sign)."""

import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def _dense(ip, ix, dt, first):
    """The (years, years) block of a CSR matrix, zeros where nothing is stored."""
    L = len(ip) - 1
    out = np.zeros((L - first, L - first))
    for r in range(first, L):
        at = slice(ip[r], ip[r + 1])
        own = ix[at] >= first
        out[r - first, ix[at][own] - first] = dt[at][own]
    return out


@pytest.mark.parametrize("form", ["zero", "subnormal", "huge", "empty"])
def test_odd_totals_and_empty_groups(form):
    torch = pytest.importorskip("torch")
    from hdfe_stream_b200 import fit
    from hdfe_stream_b200.simulate import pass0_layout, simulate_panel
    rows = pass0_layout(simulate_panel(12_000, 600, 24, spell=(4, 12), p_move=0.2, seed=4))
    first = int(sum(rows.n_levels[:-1]))
    w = np.random.default_rng(5).uniform(0.5, 2.0, len(rows.gcode))
    if form != "empty":
        group = rows.gcode == rows.gcode[len(w) // 2]
        w[group] = {"zero": 0.0, "subnormal": 1e-310, "huge": 1e307}[form]
    rows.w = w
    with np.errstate(all="ignore"):
        ref = orc.pass1(rows)
        want = _dense(*orc.build_explicit(ref), first)
    cells = fit.pass1(fit.DeviceRows.from_rows(rows))
    if form == "empty":
        # every group followed by as many empty ones as it takes for G > M
        G, M = len(cells.starts) - 1, len(cells.n)
        more = M // G + 1
        cells.starts = torch.cat([cells.starts[:1],
                                  cells.starts[1:].repeat_interleave(1 + more)]).contiguous()
        cells.group_n = torch.stack([cells.group_n] + [torch.zeros_like(cells.group_n)] * more,
                                    1).reshape(-1).contiguous()
        assert len(cells.starts) - 1 > M
    S = fit.build_s(cells)
    assert S.info["n_wide"] > 16
    got = _dense(S.indptr.cpu().numpy(), S.indices.cpu().numpy(), S.data.cpu().numpy(), first)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fine = np.isfinite(want)
    assert fine.sum() > 100 and np.array_equal(np.isfinite(got), fine)
    assert np.max(np.abs(got[fine] - want[fine])) <= 1e-12 * np.max(np.abs(want[fine]))
