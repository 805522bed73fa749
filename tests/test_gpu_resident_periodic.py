"""Periodic boxes without a boundary node take the two-kernel step, whose link kernel has nothing to do, but where
their rows are short for its tiles, and so do larger domains without force and with few boundary nodes; the same
bits either way."""
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


def _walls(nx, ny):
    return dict(nx=nx, ny=ny, periodic=(True, False), tau=0.6, collision=("trt", 0.25), accel=(1e-6, 0.0),
                kinds=[("wall", None, 0, None, None)], paint=[("rect", 0, nx - 1, 0, 0, 1), ("rect", 0, nx - 1, ny - 1, ny - 1, 1)])


def _disk(nx, ny, group=None):
    return dict(nx=nx, ny=ny, periodic=(True, True), tau=0.6, collision="bgk",
                kinds=[("wall", None, 0, group, ("circle", 0.5 * nx, 0.5 * ny, 8.3))], paint=[("shape", 1)])


def _cavity(nx, ny):
    return dict(nx=nx, ny=ny, tau=0.6, collision=("trt", 0.25), kinds=[("wall", ("const", 0.05, 0.0), 1, None, None), ("wall", None, 0, None, None)],
                paint=[("rect", 0, nx - 1, 0, 0, 2), ("rect", 0, 0, 0, ny - 1, 2), ("rect", nx - 1, nx - 1, 0, ny - 1, 2),
                       ("rect", 0, nx - 1, ny - 1, ny - 1, 1)])


@pytest.mark.parametrize("make,nx,ny,prec,resident", [
    (_walls, 500, 500, "f64", True), (_walls, 501, 500, "f64", False), (_walls, 800, 500, "f32", True), (_walls, 802, 500, "f32", False),
    (_walls, 512, 500, "f16x", False), (_disk, 800, 500, "f64", True), (_disk, 801, 500, "f64", False), (_disk, 802, 500, "f32", False),
    (lambda nx, ny: _disk(nx, ny, 0), 801, 500, "f64", True), (_cavity, 800, 799, "f64", True), (_cavity, 802, 500, "f32", False)])
def test_few_nodes(gpu, make, nx, ny, prec, resident):
    got = []
    for schedule in (None, "concurrent"):
        sim = S.product_sim(make(nx, ny), precision=prec)
        if schedule:
            sim.schedule = schedule
        sim.init((1.0, 0.01, 0.0))
        n0 = sim.launch_count()
        sim.step(36)
        got.append((sim.populations(), sim.force, sim.launch_count() - n0))
    assert (got[0][2] == 1) == resident and got[1][2] > 1
    assert np.isfinite(got[0][0]).all() and np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
