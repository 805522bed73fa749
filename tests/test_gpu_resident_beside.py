"""The resident step kernel takes most of the device for a call, so a sim leaves it alone while a batch or (a small
sim) three more sims have work in flight: their two-kernel steps overlap. The results are the same."""
import threading

import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu

LONG = 40000    # steps of a small tank: some tenths of a second


def _tank(prec="f64"):
    sim = S.product_sim(S.tunnel_like(radiating=True), precision=prec)
    sim.init((1.0, 0.02, 0.0))
    sim.vscale[1], sim.vscale[2] = 0.5, 0.002
    return sim


def _launches(sim, steps):
    n0 = sim.launch_count()
    sim.step(steps)
    return sim.launch_count() - n0


def test_fourth_sim_takes_the_two_kernel_step(gpu):
    a, b, e, c = _tank(), _tank("f32"), _tank(), _tank()
    for s in (a, b, e, c):      # (a kernel's first launch may wait for the device)
        assert _launches(s, 64) == 1
        s.synchronize()
    steps = 64
    for _ in range(5):          # (a host that is held up for as long as the others take may miss them)
        for s in (a, b, e):
            assert _launches(s, LONG) < 20                          # two others in flight at most: still resident
        n = _launches(c, 64)                                        # three others
        steps += 64
        for s in (a, b, e, c):
            s.synchronize()
        if n > 60:
            break
    assert n > 60
    assert _launches(c, 64) == 1                                    # none any more
    ref = _tank()
    ref.schedule = "concurrent"
    ref.step(steps + 64)
    assert np.array_equal(c.populations(), ref.populations())


def test_larger_sim_stays(gpu):
    small = [_tank(), _tank("f32"), _tank()]
    big = S.product_sim(S.tunnel_like(nx=702, ny=302, radiating=True))
    big.init((1.0, 0.02, 0.0))
    big.vscale[1], big.vscale[2] = 0.5, 0.002
    for s in small + [big]:
        s.step(64)
        s.synchronize()
    for s in small:
        assert _launches(s, LONG) < 20
    assert _launches(big, 64) == 1


def test_sim_beside_a_batch(gpu):
    from vortexlab_b200.batch import Batch, seeded_tunnels
    cs = seeded_tunnels(count=4, dmin=15, dmax=20, units=400.0)
    b = Batch("f32")
    for t in cs:
        b.add(t.tunnel.spec_warm(t.body), t.steps)
    b.build()
    sim = _tank()
    for _ in range(5):
        b.run_async(2000)
        n = _launches(sim, 64)
        b.wait()
        sim.synchronize()
        if n > 60:
            break
    assert n > 60
    assert _launches(sim, 64) == 1
    del b
    assert _launches(sim, 64) == 1


def test_sims_come_and_go_on_threads(gpu):
    ref = _tank()
    ref.schedule = "concurrent"
    ref.step(300)
    want = ref.populations()
    bad = []

    def work():
        for _ in range(5):
            s = _tank()
            for n in (100, 7, 193):
                s.step(n)
            if not np.array_equal(s.populations(), want):
                bad.append(1)

    ts = [threading.Thread(target=work) for _ in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
