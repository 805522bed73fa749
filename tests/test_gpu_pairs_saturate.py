"""The 16-bit fixed-point codes that saturate, in the kernels that pack two at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [48, 50])
def test_saturating_codes_match_the_one_cell_kernel(gpu, nx):
    """Populations over the whole range of the codes leave it in one step in many cells, on both sides: the groups of two
    and four cells store what the one-cell kernel stores, bit for bit."""
    V = gpu
    from vortexlab_b200.workloads import build_disk_box
    ny = 16
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    rng = np.random.default_rng(nx)
    f = w[:, None] + rng.choice([-1.0, 1.0], (9, nx * ny)) * rng.uniform(0.03, 0.13, (9, nx * ny))
    out = []
    for cells in (1, 2, 4) if nx % 4 == 0 else (1, 2):
        sim = build_disk_box(V, nx, ny, [(10.0, 8.0, 2.0)], precision="f16x")
        sim.set_cells_per_thread(cells)
        sim.schedule = "links-first"
        sim.set_populations(f.reshape(-1))
        sim.step(1)
        out.append(np.array(sim.populations()))
        sim.close()
    g = out[0].reshape(9, -1) - w[:, None]
    lim = np.where((np.arange(9) >= 1) & (np.arange(9) <= 4), 2.0 ** -18, 2.0 ** -19) * 32767
    assert (g >= lim[:, None] * 0.9999).any() and (g <= -lim[:, None]).any()      # both ends are reached
    for o in out[1:]:
        assert np.array_equal(o, out[0])
