"""fluid_grid_build beyond the one-launch sizes, where its starts come from
the sorted keys tile by tile: cells around both tile sizes (1,024 and 4,096)
and around the count at which the tile changes; cells that share a few keys,
tiles without any, and tiles with more keys than a block streams (65,536), of
one cell and of many. Against a stable argsort, exactly.
"""
import numpy as np
import pytest

from test_gpu_grid_coop import MOST, build

pytestmark = pytest.mark.gpu

LINE = 148 * 6 * 4096  # cells from which a tile is 4,096 of them


@pytest.mark.parametrize("cells,clump,spread", [
    (1, 0, 1), (1023, 0, 1), (1025, 0, 1025), (70001, MOST // 2, 900), (LINE - 1, 0, 1), (LINE, 70000, 1),
    (LINE + 4095, MOST // 2, 4096), (LINE + 4097, MOST, 3), ((1 << 24) + 3, 65537, 2)])
def test_starts_match_a_stable_sort(fcu, cells, clump, spread):
    """`clump` positions in the `spread` cells from the middle on, the rest anywhere."""
    import torch
    n = MOST + 1
    rng = np.random.default_rng(cells)
    want_keys = rng.integers(0, cells, n)
    want_keys[rng.permutation(n)[:clump]] = cells // 2 + rng.integers(0, spread, clump)
    want_keys = np.minimum(want_keys, cells - 1)
    pos = torch.zeros((n, 4), device="cuda")
    # x below 2^24: exact in 32 bits; the last cells by their clamp
    pos[:, 0] = torch.from_numpy(want_keys.astype(np.float32)).cuda()
    want_keys = np.minimum(want_keys.astype(np.float32).astype(np.int64), cells - 1)
    keys, starts, perm = build(fcu, torch, pos, (cells, 1, 1))
    counts = np.bincount(want_keys, minlength=cells)
    assert np.array_equal(keys[:n], want_keys) and np.all(keys[n:] == -5)
    assert starts[0] == 0 and np.array_equal(starts[1:-8], np.cumsum(counts)) and np.all(starts[-8:] == -7)
    assert np.array_equal(perm[:n], np.argsort(want_keys, kind="stable")) and np.all(perm[n:] == -9)
