"""The resident step kernel with many boundary nodes: the tables of a block in its shared memory, or, where they
do not fit (FP64, a random half of the cells solid), in global memory. The same bits as the two-kernel step."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


def _disks(nx, ny):
    from vortexlab_b200.workloads import disk_field
    return disk_field(nx, ny, seed=3, fraction=0.25, rmin=1.5, rmax=3.0)


def _cells(nx, ny):
    g = np.random.default_rng(4)
    y, x = np.nonzero(g.random((ny - 2, nx - 2)) < 0.5)
    return np.stack([x + 1.0, y + 1.0, np.full(x.size, 0.6)], axis=1)


def _box(nx, ny, disks, group):
    d = S.disk_box(nx, ny, disks)
    d["kinds"] = [("wall", None, 0, group, ("disks", disks))]
    return d


def _run(d, prec, schedule, calls):
    sim = S.product_sim(d, precision=prec)
    if schedule:
        sim.schedule = schedule
    sim.init((1.0, 0.03, 0.01))
    sim.record(sum(calls))
    n0 = sim.launch_count()
    for n in calls:
        sim.step(n)
    return sim.populations(), sim.history(), sim.launch_count() - n0


@pytest.mark.parametrize("prec", ["f64", "f32", "f16x"])
@pytest.mark.parametrize("make,nx,ny", [(_disks, 640, 400), (_cells, 350, 370)])
def test_many_boundary_nodes(gpu, make, nx, ny, prec):
    d = _box(nx, ny, make(nx, ny), None)
    f0, h0, n0 = _run(d, prec, "concurrent", [5, 36])
    f1, h1, n1 = _run(d, prec, None, [5, 36])
    assert n1 == 2 < n0
    assert np.isfinite(f0).all() and np.array_equal(f0, f1) and np.array_equal(h0, h1)


def test_force_on_many_nodes_takes_the_two_kernel_step(gpu):
    """The force sums of the resident kernel are one block's work: with force on most of 60,000 boundary nodes it was
    three times as slow as the two-kernel step."""
    d = _box(640, 400, _disks(640, 400), 0)
    f0, h0, n0 = _run(d, "f64", "concurrent", [5, 36])
    f1, h1, n1 = _run(d, "f64", None, [5, 36])
    assert n1 == n0 and np.array_equal(f0, f1) and np.array_equal(h0, h1) and np.abs(h0).max() > 0
