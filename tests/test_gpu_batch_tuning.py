"""The autotuner's choice where a block size reaches no kernel: in a batch small
enough for the lane-shared sweeps every candidate times the same launch, so the
choice stays the default instead of following the clock's noise.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_small_batches_keep_the_default(fcu, wl):
    cfgs = wl.batched_boxes(fcu, nboxes=3, seed=5, lo=500, hi=2000)
    batch = fcu.Batch(cfgs)
    steps = wl.batched_frame_steps(fcu, 3, frames=1, substeps=2, seed=9)
    batch.run(steps)
    for _ in range(6):
        chosen, ms = batch.autotune(steps[0])
        assert (ms > 0).all()
        integrate = chosen.pop("integrate")
        assert set(chosen.values()) == {128} and integrate in (64, 128, 256), chosen
