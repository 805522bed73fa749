"""Sim.vorticity on the device against the oracle's (FP64 differences rounded once to FP32): equal bit for bit on
domains with solids in every position, one-sided at edges; repeated calls between other field reads, which share
the sim's scratch memory, from two threads."""
import threading

import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


def _domains():
    from vortexlab_b200.workloads import disk_field
    return {"disks": S.disk_box(300, 140, disk_field(300, 140, seed=5)), "tunnel": S.tunnel_like(radiating=True),
            "walls": S.tunnel_like(nx=121, radiating=False), "no_walls": S.periodic_box(3, 5, collision="bgk")}


@pytest.mark.parametrize("name", ["disks", "tunnel", "walls", "no_walls"])
def test_vorticity_against_oracle(gpu, O, name):
    d = _domains()[name]
    sim, osim = S.product_sim(d), S.oracle_sim(d)
    f = S.swirl(d["nx"], d["ny"])
    sim.init(f)
    osim.init(f)
    for steps in (0, 7):
        sim.step(steps)
        if steps:
            osim.step(steps)
        assert np.array_equal(sim.vorticity(), osim.vorticity())


def test_field_reads_share_scratch_memory(gpu):
    d = _domains()["tunnel"]
    sim = S.product_sim(d, precision="f32")
    sim.init(S.swirl(d["nx"], d["ny"]))
    sim.step(20)
    want = (sim.vorticity(), sim.macros_field(), sim.populations())
    bad = []

    def read(k):
        for i in range(30):
            if (i + k) % 3 == 0 and not np.array_equal(sim.vorticity(), want[0]):
                bad.append("vorticity")
            if (i + k) % 3 == 1 and not all(np.array_equal(a, b) for a, b in zip(sim.macros_field(), want[1])):
                bad.append("macros")
            if (i + k) % 3 == 2 and not np.array_equal(sim.populations(), want[2]):
                bad.append("populations")

    ts = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
