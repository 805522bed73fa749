"""The batched step in one launch (schedule "concurrent"): outlets of fewer nodes than a block, just under and over one
and two blocks, one and many tunnels, whole and partial graphs, in every storage format."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32", "f16s", "f16c", "f16x"])
@pytest.mark.parametrize("sizes", [[3], [25, 26, 12], [51, 52, 7, 13]])
@pytest.mark.parametrize("steps", [5, 70])
def test_one_launch_matches_two(gpu, prec, sizes, steps):
    """Populations and forces, bit for bit, against the link kernel and then the bulk kernel; also in the one-cell form."""
    from vortexlab_b200.batch import Batch, seeded_tunnels
    cases = [seeded_tunnels(seed=77 + d, count=1, dmin=d, dmax=d, re=(40.0, 120.0), units=1.0, precision=prec)[0] for d in sizes]
    want = None
    for sched, cells in (("links-first", None), ("concurrent", None), ("concurrent", 1)):
        if cells and prec == "f64":
            continue
        b = Batch(prec)
        for k, c in enumerate(cases):
            b.add(c.tunnel.spec_warm(c.body), steps + 3 * k)      # they end one after another
        b.build()
        b.schedule = sched
        if cells:
            b.set_cells_per_thread(cells)
        b.run()
        got = [(b.status(k)[0], b.state_hash(k), b.force_history(k)) for k in range(len(sizes))]
        b.close()
        if want is None:
            want = got
        for (t, h, f), (t0, h0, f0) in zip(got, want):
            assert t == t0 and h == h0 and np.isfinite(f).all() and np.array_equal(f, f0), (sched, cells)
