"""A vorticity frame takes no more device memory than the fields it is formed from."""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


def test_vorticity_where_the_fields_fit(gpu):
    import torch
    V = gpu
    nx, ny = 4096, 1024                     # 96 MiB of fields, 112 with a frame beside them: neither is kept
    sim = S.product_sim(S.periodic_box(nx, ny, collision="bgk"), precision="f16x")
    sim.init((1.0, 0.05, 0.0))
    sim.step(3)
    want = sim.vorticity()
    rho, ux, uy = sim.macros_field()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (104 << 20), dtype=torch.uint8, device="cuda")
    try:
        fields = sim.macros_field()
        got = sim.vorticity()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.array_equal(got, want) and np.array_equal(fields[1], ux)
