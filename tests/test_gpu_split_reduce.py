"""The sum of a split product's parts: every number of parts around the batches that the kernel loads."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 7, 8, 9, 15, 16, 17, 24, 31, 47, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 192, 193, 296])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_every_part_is_added_once(gpu, splits, accumulate):
    """Small whole numbers: every sum is exact in FP32, so a part left out or added twice changes the result."""
    import torch
    V = gpu
    M, N, K = 32, 32, 512 * splits            # a part is eight blocks of 64
    g = torch.Generator(device="cuda").manual_seed(splits)
    a = torch.randint(-2, 3, (M, K), generator=g, device="cuda").float()
    b = torch.randint(-2, 3, (N, K), generator=g, device="cuda").float()
    out = torch.randint(-50, 51, (M, N), generator=g, device="cuda").float()
    want = (a.double() @ b.double().t() + accumulate * out.double()).float()
    a, b = a.bfloat16(), b.bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = V.lib.vl_nn_gemm_bf16(C.c_void_p(a.data_ptr()), K, C.c_void_p(b.data_ptr()), K, M, N, K, C.c_void_p(out.data_ptr()), N,
                               C.cast(C.c_void_p(0), C.POINTER(C.c_float)), accumulate, 32,
                               C.cast(C.c_void_p(err.data_ptr()), C.POINTER(C.c_int)), None)
    assert rc == 0 and int(err.item()) == 0
    assert torch.equal(out, want)
