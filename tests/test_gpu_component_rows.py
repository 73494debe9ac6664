"""Rows per component (`pair_components`): counts carried along a thread's
walk and added per warp and label, against a bincount over networks made of
disjoint blocks -- one giant block, blocks that alternate within a warp, and
more pairs than the grid has threads."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [[1], [31, 1, 1], [1] * 70, [200_000, 5, 120_000, 1]])
def test_rows_per_component(blocks):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from hdfe_stream_b200.connected import pair_components
    of = np.repeat(np.arange(len(blocks)), blocks)      # each worker's block
    a = np.repeat(np.arange(len(of)), 3)                # two rows at the block's first firm,
    b = 2 * of[a] + (np.arange(len(a)) % 3 == 2)        # one at its second
    t = lambda x: torch.as_tensor(x.astype(np.int32), device="cuda")
    label, rows, info = pair_components(t(a), t(b), len(of), 2 * len(blocks))
    assert info["components"] == len(blocks)
    assert sorted(rows) == sorted(3 * np.asarray(blocks))
    label = label.cpu().numpy()
    assert all(rows[c] == np.count_nonzero(label[a] == c) for c in range(len(rows)))
