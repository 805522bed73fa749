"""A wait of the resident step kernel that runs out: reported by every call that steps the sim or reads its state,
over once the sim is started again. The blocks wait for an arrival that none makes (vl_sim_test_stall); the waits are
bounded."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,steps", [("f64", 8), ("f32", 3 * 4096), ("f16x", 5)])
def test_stalled_step_is_reported_and_init_starts_again(gpu, prec, steps):
    V = gpu
    d = S.tunnel_like(radiating=True)
    sim = S.product_sim(d, precision=prec)

    def run():
        sim.init((1.0, 0.02, 0.0))
        sim.record(60)
        sim.vscale[1], sim.vscale[2] = 0.5, 0.002
        sim.step(60)
        return sim.populations(), sim.history(), sim.t

    want = run()
    V._lib.check(V.lib.vl_sim_test_stall(sim._h, steps))
    reads = [lambda: sim.synchronize(), lambda: sim.populations(), lambda: sim.macros_field(), lambda: sim.vorticity(),
             lambda: sim.total_mass(), lambda: sim.max_speed(), lambda: sim.macros(5, 5), lambda: sim.force, lambda: sim.t,
             lambda: sim.history(), lambda: sim.status(), lambda: sim.state_hash(), lambda: sim.last_step_ms(),
             lambda: sim.step(1), lambda: sim.step(64), lambda: sim.set_populations(want[0])]
    for k, read in enumerate(reads):
        with pytest.raises(V.VortexError, match="gave up waiting"):
            read()
            pytest.fail(f"call {k} did not report the stalled step")
    got = run()
    assert np.isfinite(want[0]).all()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2] == want[2]


def test_other_sims_do_not_stall(gpu):
    V = gpu
    sim = S.product_sim(S.tunnel_like(nx=1400, ny=700, radiating=True))     # two buffers larger than the L2
    assert V.lib.vl_sim_test_stall(sim._h, 8) < 0
    sim.step(8)
    sim.synchronize()


@pytest.mark.parametrize("before", [0, 5])
def test_refused_launch_takes_the_two_kernel_step(gpu, before):
    """A cooperative launch that the device refuses (here for its number of blocks): the same steps by two kernels."""
    V = gpu
    got = []
    for refuse in (False, True):
        sim = S.product_sim(S.tunnel_like(radiating=True))
        sim.init((1.0, 0.02, 0.0))
        sim.record(120)
        sim.vscale[1], sim.vscale[2] = 0.5, 0.002
        if before:
            sim.step(before)
        if refuse:
            V._lib.check(V.lib.vl_sim_test_refused(sim._h, 70))
        else:
            sim.step(70)
        n0 = sim.launch_count()
        sim.step(40)
        assert (sim.launch_count() - n0 > 40) == refuse
        assert sim.last_step_ms() > 0
        got.append((sim.populations(), sim.history(), sim.t))
    assert got[0][2] == got[1][2] == 110 + before
    assert np.isfinite(got[0][0]).all()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
