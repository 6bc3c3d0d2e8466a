"""fluid_grid_build on the default stream while a context of a slice of the SMs
is current: the same starts and permutation as with the whole GPU.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side", [(5000, 16), (200003, 50)])
def test_the_default_stream_of_a_slice_builds_the_same_grid(fcu, n, side):
    import torch
    d = pytest.importorskip("cuda.bindings.driver")

    def ok(out):
        assert out[0] == d.CUresult.CUDA_SUCCESS, out[0]
        return out[1:]

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
    dev, = ok(d.cuDeviceGet(0))
    whole, = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(d.cuDevSmResourceSplitByCount(1, whole, 0, 24))
    desc, = ok(d.cuDevResourceGenerateDesc([groups[0]], 1))
    green, = ok(d.cuGreenCtxCreate(desc, dev, d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    ctx, = ok(d.cuCtxFromGreenCtx(green))
    ok(d.cuCtxPushCurrent(ctx))
    try:
        fcu.grid_build_device(d_pos.data_ptr(), n, g, 0, starts.data_ptr(), perm.data_ptr(), ws.data_ptr(), bytes_, 0)
        ok(d.cuCtxSynchronize())
    finally:
        ok(d.cuCtxPopCurrent())
    assert fcu.grid_build_status(ws.data_ptr(), n, g) == fcu.OK
    assert np.array_equal(perm.cpu().numpy(), np.argsort(key, kind="stable"))
    counts = np.bincount(key, minlength=side ** 3)
    assert np.array_equal(starts.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    ok(d.cuGreenCtxDestroy(green))
