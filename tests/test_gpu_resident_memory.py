"""A sim whose own buffers fit the device and the resident step kernel's tables do not is built all the same, and
takes the two-kernel step."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


def test_sim_is_built_without_room_for_the_resident_tables(gpu):
    import torch
    from vortexlab_b200.workloads import disk_field
    V = gpu
    disks = disk_field(640, 400, seed=3, fraction=0.25, rmin=1.5, rmax=3.0)
    d = S.disk_box(640, 400, disks)
    d["kinds"] = [("wall", None, 0, None, ("disks", disks))]

    def run(sim):
        sim.init((1.0, 0.03, 0.01))
        n0 = sim.launch_count()
        sim.step(40)
        return sim.populations(), sim.launch_count() - n0

    want, launches = run(S.product_sim(d, precision="f32"))
    assert launches == 1
    torch.cuda.empty_cache()
    step = 2 << 20
    seen = set()
    for room in range(step, 96 * step, step):
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - room, dtype=torch.uint8, device="cuda")
        try:
            sim = S.product_sim(d, precision="f32")
        except V.VortexError:
            sim = None
        del hog
        torch.cuda.empty_cache()
        if sim is None:
            seen.add("refused")
            continue
        got, launches = run(sim)
        assert np.array_equal(got, want)
        seen.add("two kernels" if launches > 1 else "resident")
        if launches == 1:
            break
    assert seen == {"refused", "two kernels", "resident"}
