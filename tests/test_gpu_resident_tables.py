"""The resident step kernel with so many boundary nodes that a block's tables stay in global memory (FP64), and
with nearly as many in its shared memory (FP32): the same bits as the two-kernel step."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32", "f16x"])
def test_dense_disks(gpu, prec):
    from vortexlab_b200.workloads import disk_field
    d = S.disk_box(640, 400, disk_field(640, 400, seed=3, fraction=0.25, rmin=1.5, rmax=3.0))
    got = []
    for schedule in (None, "concurrent"):
        sim = S.product_sim(d, precision=prec)
        if schedule:
            sim.schedule = schedule
        sim.init((1.0, 0.03, 0.01))
        sim.record(41)
        n0 = sim.launch_count()
        for n in (5, 36):
            sim.step(n)
        got.append((sim.populations(), sim.history(), sim.force))
        assert (sim.launch_count() - n0 == 2) == (schedule is None)
    assert np.isfinite(got[0][0]).all() and np.abs(got[0][1]).max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)
