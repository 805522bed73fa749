"""FP64 batches around the number of tiles at which the one-launch step changes its block bound: the populations and force
histories of the same tunnels stepped by two kernels one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(15,), (16, 19), (40, 40), (15, 24, 31, 40), (30, 40, 44), (40, 40, 40, 40)])
def test_one_launch_step(gpu, sizes):
    from vortexlab_b200.batch import Batch, seeded_tunnels
    got = []
    for schedule in ("concurrent", "links-first"):
        b = Batch("f64")
        for k, d in enumerate(sizes):
            c = seeded_tunnels(seed=77 + k, count=1, dmin=d, dmax=d, re=(60.0, 120.0), units=40.0, precision="f64")[0]
            b.add(c.tunnel.spec_warm(c.body), 75)
        b.build()
        b.schedule = schedule
        b.run(40)
        b.run()
        got.append([(b.populations(k), b.force_history(k)) for k in range(len(sizes))])
    for (f0, h0), (f1, h1) in zip(*got):
        assert np.isfinite(f0).all() and np.array_equal(f0, f1) and np.array_equal(h0, h1)
