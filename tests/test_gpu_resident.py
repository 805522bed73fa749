"""The resident step kernel (many steps of a small domain in one launch) against the two-kernel step.

Every population, force, outlet offset, record and pressure drop it computes follows the two-kernel
step's expressions in its order, so all results must be equal bit for bit: on every link rule and
storage format, for numbers of steps around its smallest call, odd and even (the buffers swap), with
controls set between calls, mixed with calls too short for it, and beside another sim's kernel.
"""
import threading

import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


def _domains():
    from vortexlab_b200.workloads import disk_field
    return {
        "disk_box_640x200": S.disk_box(640, 200, disk_field(640, 200, seed=11)),   # no outlet, body across chunks
        "tunnel_like": S.tunnel_like(radiating=True),                              # rows end inside a warp
        "tunnel_walls_121": S.tunnel_like(nx=121, radiating=False),                # odd rows: one cell per thread
        "tunnel_tall": S.tunnel_like(nx=67, ny=300, radiating=True),               # more outlet nodes than 256
        "forced": S.poiseuille(rows=16, q=0.8, collision=("trt", 0.25)),
        "three_wide": S.periodic_box(3, 37, collision="bgk"),                      # the smallest row, no boundary
    }


def _run(d, prec, schedule, calls):
    sim = S.product_sim(d, precision=prec)
    if schedule:
        sim.schedule = schedule
    if d.get("periodic", (False, False)) == (True, True):
        sim.init(S.swirl(d["nx"], d["ny"]))
    else:
        sim.init((1.0, 0.02, 0.0))
    sim.record(sum(calls))
    out = []
    for k, n in enumerate(calls):
        if not d.get("accel"):
            sim.vscale[1] = 0.5 + 0.05 * k
            sim.vscale[2] = 0.002 * np.sin(0.3 * k)
            if k != 2:
                sim.outflow_target = 0.05 * (0.5 + 0.05 * k)
            else:
                sim.outflow_target = None
        sim.step(n)
        out.append((sim.t, sim.force, sim.outlet_density_offset, sim.status()))
    return sim.populations(), sim.history(), out, sim.launch_count()


@pytest.mark.parametrize("prec", ["f64", "f32", "f16s", "f16c", "f16x"])
@pytest.mark.parametrize("name", ["disk_box_640x200", "tunnel_like", "tunnel_walls_121", "tunnel_tall", "forced", "three_wide"])
def test_matches_the_two_kernel_step(gpu, name, prec):
    d = _domains()[name]
    calls = [4, 5, 37, 3, 64, 1, 2, 33]
    f0, h0, o0, n0 = _run(d, prec, "concurrent", calls)
    f1, h1, o1, n1 = _run(d, prec, None, calls)
    assert n1 < n0 / 4, "the resident kernel did not run"
    assert np.isfinite(f0).all()
    assert np.array_equal(f0, f1) and np.array_equal(h0, h1)
    for a, b in zip(o0, o1):
        assert a[0] == b[0] and np.array_equal(a[1], b[1]) and a[2] == b[2] and a[3] == b[3]


def test_several_launches_per_call_and_the_probe(gpu):
    """More steps than one launch takes, with the pressure probe recorded at every step."""
    V = gpu
    res = []
    for schedule in (None, "concurrent"):
        r = V.cylinder.rig(V.cylinder.Setup(n=10), 60.0, 2.0)
        if schedule:
            r.ch.sim.schedule = schedule
        res.append(V.cylinder.run_record(r, 4096 + 7) + (r.ch.sim.populations(), r.ch.sim.vscale[1], r.ch.sim.t))
    for a, b in zip(*res):
        assert np.array_equal(a, b)


def test_cells_per_thread_and_autotune_keep_the_results(gpu):
    d = _domains()["tunnel_like"]
    ref = _run(d, "f32", "concurrent", [50, 50])
    sim = S.product_sim(d, precision="f32")
    sim.set_cells_per_thread(1)
    sim.init((1.0, 0.02, 0.0))
    sim.record(100)
    for k in range(2):
        sim.vscale[1] = 0.5 + 0.05 * k
        sim.vscale[2] = 0.002 * np.sin(0.3 * k)
        sim.outflow_target = 0.05 * (0.5 + 0.05 * k)
        sim.step(50)
        sim.set_cells_per_thread(2)
        sim.autotune(2)
    assert np.array_equal(sim.populations(), ref[0]) and np.array_equal(sim.history(), ref[1])


def test_divergence_is_marked_at_the_same_step(gpu):
    """Non-finite forces: the same first step as the two-kernel step's."""
    d = _domains()["tunnel_like"]
    got = []
    for schedule in (None, "links-first"):
        sim = S.product_sim(d)
        if schedule:
            sim.schedule = schedule
        sim.init((1.0, 0.02, 0.0))
        f = sim.populations().copy()
        f[:, d["ny"] // 2, 5] = np.nan
        sim.set_populations(f)
        sim.step(120)
        got.append(sim.status())
    assert got[0] == got[1] and got[0][0]


def test_two_sims_on_two_threads(gpu):
    """Two sims' kernels on their own streams, from two host threads."""
    d = _domains()["tunnel_like"]
    ref = _run(d, "f64", "concurrent", [200, 200])
    out = [None, None]

    def work(k):
        out[k] = _run(d, "f64", None, [200, 200])

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for o in out:
        assert np.array_equal(o[0], ref[0]) and np.array_equal(o[1], ref[1])
