"""The body splat at every lane count its rule chooses, by the quad's columns
and the particle count (under 5 columns, up to 7.3, 10, 24 and beyond, below
and from 100,000 particles), against the oracle bit for bit.
"""
import pytest

from test_gpu_field import oracle_field
from test_gpu_step import assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(11, 9, 7), (47, 46, 47)], ids=["693", "101614"])
def sim(request, fcu, wl):
    block = request.param
    s = fcu.Sim(wl.box_config(fcu, block, tuple(0.01 * k for k in block), 0.005, solve=fcu.SOLVE_FIXED))
    s.run([fcu.make_step(force=(0.2, -9.81, 0.1), dt=1e-3, v_clamp=2.0)] * 2)
    return s


@pytest.mark.parametrize("lens", [0, 4])
@pytest.mark.parametrize("columns", [3.5, 4.9, 5.2, 7.2, 7.6, 9.9, 10.3, 23.5, 24.6, 40.0])
def test_splat_matches_the_oracle(orc, sim, columns, lens):
    # the width that gives a quad about that many columns
    w = max(1, round((columns - 3.0) * sim.params.tracer_e[0] / (1.5 * sim.params.h)))
    h = max(1, w // 2 + 3)
    sim.field_splat(w, h, keep=0.0, lens=lens, lo=0.0, hi=0.5)
    field, _ = sim.field_read()
    assert field[..., 0].max() > 0.0
    assert_same_bits(field, oracle_field(orc, sim, w, h, 0.0, lens, 0.0, 0.5, None), f"{w} x {h}")
