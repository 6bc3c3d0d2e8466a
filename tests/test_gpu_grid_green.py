"""fluid_grid_build on a stream that may use only some of the SMs (a green
context's): where the one-launch build's blocks would not all be resident the
digit passes answer, where they would (a small input) the one launch does, and
either way the same starts and permutation, also replayed from a graph.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def slice_stream():
    import torch
    d = pytest.importorskip("cuda.bindings.driver")

    def ok(out):
        assert out[0] == d.CUresult.CUDA_SUCCESS, out[0]
        return out[1:]

    torch.zeros(1, device="cuda")
    dev, = ok(d.cuDeviceGet(0))
    whole, = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(d.cuDevSmResourceSplitByCount(1, whole, 0, 24))
    assert 24 <= groups[0].sm.smCount < 148
    desc, = ok(d.cuDevResourceGenerateDesc([groups[0]], 1))
    ctx, = ok(d.cuGreenCtxCreate(desc, dev, d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream, = ok(d.cuGreenCtxStreamCreate(ctx, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(stream))
    torch.cuda.synchronize()
    ok(d.cuStreamDestroy(stream))
    ok(d.cuGreenCtxDestroy(ctx))


@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.parametrize("n,side", [(5000, 16), (200003, 50), (148 * 8192, 100)])
def test_a_slice_of_the_gpu_builds_the_same_grid(fcu, slice_stream, n, side, capture):
    import torch
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, side, (n, 3))
    cell = pos[:, :3].astype(np.int64)
    key = (cell[:, 2] * side + cell[:, 1]) * side + cell[:, 0]
    g = fcu.FluidGrid()
    g.cell = 1.0
    g.dims[:] = [side] * 3
    d_pos = torch.from_numpy(pos).cuda()
    bytes_ = fcu.grid_workspace_bytes(n, g)
    ws = torch.empty(bytes_, dtype=torch.uint8, device="cuda")
    starts = torch.full((side ** 3 + 1,), -1, dtype=torch.int32, device="cuda")
    perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def build():
        fcu.grid_build_device(d_pos.data_ptr(), n, g, 0, starts.data_ptr(), perm.data_ptr(), ws.data_ptr(), bytes_,
                              slice_stream.cuda_stream)

    with torch.cuda.stream(slice_stream):
        if capture:
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin(capture_error_mode="thread_local")
            build()
            graph.capture_end()
            graph.replay()
        else:
            build()
    slice_stream.synchronize()
    assert fcu.grid_build_status(ws.data_ptr(), n, g) == fcu.OK
    assert np.array_equal(perm.cpu().numpy(), np.argsort(key, kind="stable"))
    counts = np.bincount(key, minlength=side ** 3)
    assert np.array_equal(starts.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
