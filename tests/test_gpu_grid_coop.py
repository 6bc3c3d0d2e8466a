"""fluid_grid_build where its path changes: one cooperative launch up to
148 x 8,192 positions, digit passes beyond; digits of four to eight bits in
one to three passes; pieces with and without a ragged end; more blocks for
the cells than the positions fill. Starts and permutation against a stable
argsort, exactly, in buffers whose ends are checked; and the same build
replayed from a CUDA graph.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOST = 148 * 8192


def build(fcu, torch, pos, dims, capture=False):
    n, cells = pos.shape[0], dims[0] * dims[1] * dims[2]
    g = fcu.FluidGrid()
    g.cell = 1.0
    g.dims[:] = dims
    bytes_ = fcu.grid_workspace_bytes(n, g)
    ws = torch.full((bytes_,), 0x5A, dtype=torch.uint8, device="cuda")
    starts = torch.full((cells + 9,), -7, dtype=torch.int32, device="cuda")
    perm = torch.full((n + 8,), -9, dtype=torch.int32, device="cuda")
    keys = torch.full((n + 8,), -5, dtype=torch.int32, device="cuda")

    def run():
        fcu.grid_build_device(pos.data_ptr(), n, g, keys.data_ptr(), starts.data_ptr(), perm.data_ptr(),
                              ws.data_ptr(), bytes_, torch.cuda.current_stream().cuda_stream)

    run()
    if capture:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        ws.fill_(0x33)
        for b in (starts, perm, keys):
            b[:-8] = -1
        graph.replay()
    torch.cuda.synchronize()
    assert fcu.grid_build_status(ws.data_ptr(), n, g) == fcu.OK
    return [b.cpu().numpy() for b in (keys, starts, perm)]


@pytest.mark.parametrize("n,dims,clump", [
    (1, (1, 1, 1), 0), (31, (4, 4, 1), 0), (1023, (17, 1, 1), 0), (1024, (16, 16, 1), 500),
    (1025, (257, 1, 1), 0), (8193, (40, 41, 10), 8000), (20011, (24, 24, 24), 0),
    (40000, (128, 64, 64), 20000), (300007, (64, 33, 31), 290000), (MOST, (100, 100, 100), 0),
    (MOST + 1, (100, 100, 100), 0)])
def test_builds_match_a_stable_sort(fcu, n, dims, clump):
    import torch
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(-0.5, np.array(dims) + 0.5, (n, 3))  # some outside: clamped
    at = rng.permutation(n)[:clump]
    pos[at, :3] = np.array(dims) * 0.5
    cell = np.minimum(np.maximum(pos[:, :3], 0).astype(np.int64), np.array(dims) - 1)
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
