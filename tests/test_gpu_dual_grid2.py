"""The dual grid through a two-level rank bitmap against the plain bitmap and the sorted keys: the same
dual centres, cubes and counts for leaf cells of strides 1 to 128 (faces of strides from 32 on are found
from the centres that exist), in boxes whose corner lies off every lattice, at one, two and four samples
a side, with levels that are empty."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def random_leaves(levels, split, seed, shift):
    """Disjoint leaf cells: coarsest cells split at random down to stride 1."""
    rng = np.random.default_rng(seed)
    s = 2 ** (levels - 1)
    cells = np.stack(np.meshgrid(np.arange(3), np.arange(2), np.arange(2), indexing="ij"), -1).reshape(-1, 3) * s + shift * s
    out = {}
    octants = np.stack(np.meshgrid([0, 1], [0, 1], [0, 1], indexing="ij"), -1).reshape(-1, 3)
    for d in range(levels - 1, -1, -1):
        cut = rng.random(len(cells)) < (split if d > 0 else 0.0)
        leaves = cells[~cut]
        order = np.lexsort(leaves.T[::-1])
        out[d] = torch.from_numpy(leaves[order].astype(np.int32)).to(DEV).reshape(-1, 3).contiguous()
        cells = (cells[cut][:, None] + octants[None] * (2 ** d // 2)).reshape(-1, 3)
    return out


@pytest.mark.parametrize("levels,split,n_up,shift", [(1, 0.0, 2, 0), (3, 0.5, 1, -1), (6, 0.45, 2, -2), (7, 0.4, 4, 1),
                                                     (8, 0.4, 2, -1), (8, 0.4, 1, 3), (8, -0.4, 2, 0)])
def test_two_level_equals_plain_and_sorted(levels, split, n_up, shift):
    from jspsr.core.pipeline import DualMesher
    base = random_leaves(levels, abs(split), levels * 10 + n_up, np.array([shift, -shift, 2 * shift]))
    if split < 0:
        base[2] = base[2][:0]                                # a level without leaves
    got = []
    for plain, two in ((1 << 27, 0), (0, 1 << 27), (0, 0)):
        m = DualMesher()
        m.levels = [SimpleNamespace(stride=2 ** d) for d in range(levels)]
        m.vs, m.dev, m.dual_grid_max_words, m.dual_grid2_max_words = 1.0 / 64, DEV, plain, two
        v, f = m.mesh_from_leaves(dict(base), levels, n_up, lambda p: torch.sin(97.0 * p.sum(1) + 1.0))
        got.append((m.mesh_info["cnt"], m.mesh_info["acc_ids"], f, v))
    assert int((got[0][0] == 8).sum()) > 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a, b)
