"""The body splat at field sizes on both sides of each lane count it chooses
by (quads of 4, 8 and more columns, and wider than a particle's 16 lanes),
with and without the lens, against the oracle bit for bit."""
import pytest

from test_gpu_field import oracle_field, settled_sim
from test_gpu_step import assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,lens", [(1, 1, 4), (3, 5, 0), (32, 64, 4), (45, 20, 0), (97, 201, 4), (295, 639, 3),
                                      (640, 33, 0)])
def test_splat_matches_the_oracle(fcu, orc, w, h, lens):
    sim = settled_sim(fcu, 2)
    lo, hi = (500.0, 1000.0) if lens == 3 else (0.0, 0.5)
    sim.field_splat(w, h, keep=0.0, lens=lens, lo=lo, hi=hi)
    field, _ = sim.field_read()
    assert_same_bits(field, oracle_field(orc, sim, w, h, 0.0, lens, lo, hi, None), f"{w} x {h}")
