"""Periodic boxes without a boundary node take the two-kernel step, whose link kernel has nothing to do, but where
their rows are short for its tiles; the same bits either way."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,prec,resident", [
    (50, 50, "f64", False), (32, 40, "f64", False), (31, 40, "f64", True), (3, 100, "f32", True), (33, 64, "f32", False),
    (50, 50, "f32", False), (100, 2000, "f32", True), (100, 1999, "f32", False), (104, 2000, "f32", False), (200, 2100, "f16x", True),
    (208, 2100, "f16x", False), (102, 2001, "f16x", True), (106, 2001, "f16x", False), (801, 99, "f16x", False)])
def test_route(gpu, nx, ny, prec, resident):
    got = []
    for schedule in (None, "concurrent"):
        sim = S.product_sim(S.periodic_box(nx, ny, collision="bgk"), precision=prec)
        if schedule:
            sim.schedule = schedule
        sim.init(S.swirl(nx, ny))
        n0 = sim.launch_count()
        sim.step(40)
        got.append((sim.populations(), sim.launch_count() - n0))
    assert (got[0][1] == 1) == resident and got[1][1] > 1
    assert np.isfinite(got[0][0]).all() and np.array_equal(got[0][0], got[1][0])
