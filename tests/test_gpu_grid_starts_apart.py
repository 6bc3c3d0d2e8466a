"""The one-launch grid build around the cell count from which the starts are a
launch of their own (400,000 cells), with three digit passes and with four, in
any order, clumped and all in one cell, and replayed from a graph: starts and
permutation against a stable argsort, exactly, in buffers whose ends are
checked.
"""
import numpy as np
import pytest

from test_gpu_grid_coop import MOST, build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dims,clump", [
    (33, (400000, 1, 1), 0), (20011, (400000, 1, 1), 0), (20011, (400001, 1, 1), 15000), (1, (800, 600, 1), 0),
    (150001, (100, 100, 41), 150001), (300007, (260, 256, 256), 100000), (MOST, (128, 127, 126), 0),
    (MOST, (73, 75, 77), 1000000)])
def test_builds_match_a_stable_sort(fcu, n, dims, clump):
    import torch
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, np.array(dims), (n, 3))
    pos[rng.permutation(n)[:clump], :3] = np.array(dims) * 0.5
    cell = np.minimum(pos[:, :3].astype(np.int64), np.array(dims) - 1)
    want_keys = (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
    want_perm = np.argsort(want_keys, kind="stable")
    counts = np.bincount(want_keys, minlength=dims[0] * dims[1] * dims[2])
    want_starts = np.concatenate([[0], np.cumsum(counts)])
    d_pos = torch.from_numpy(pos).cuda()
    for capture in (False, True):
        keys, starts, perm = build(fcu, torch, d_pos, dims, capture)
        assert np.array_equal(keys[:n], want_keys) and np.all(keys[n:] == -5)
        assert np.array_equal(starts[:-8], want_starts) and np.all(starts[-8:] == -7)
        assert np.array_equal(perm[:n], want_perm) and np.all(perm[n:] == -9)
