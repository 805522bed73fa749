"""A schedule that does not exist is refused and changes nothing."""
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-1, 4, 99])
def test_refused_schedule_leaves_the_resident_step(gpu, bad):
    V = gpu
    sim = S.product_sim(S.tunnel_like(radiating=True))
    sim.init((1.0, 0.02, 0.0))
    sim.step(64)
    n0 = sim.launch_count()
    assert V.lib.vl_sim_set_schedule(sim._h, bad) < 0
    sim.step(64)
    assert sim.launch_count() - n0 == 1
    sim.schedule = "concurrent"
    n0 = sim.launch_count()
    sim.step(64)
    assert sim.launch_count() - n0 > 1
