"""A convolution of so many channels that the bytes of its weights do not fit 31 bits: the shared-memory rule of the
row kernel must not take it. Against im2col and the GEMM."""
import pytest

pytestmark = pytest.mark.gpu


def test_half_a_million_channels(gpu):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    C, N = 466048, 256
    kp = 9 * C
    assert 9 * C * N * 2 > 2 ** 31 - 1 and kp % 64 == 0
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(1, 1, 1, C, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.empty(N, kp, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    b = torch.randn(N, generator=g, device="cuda")
    cols = torch.zeros(1, kp, dtype=torch.bfloat16, device="cuda")
    want, got = torch.zeros(1, N, device="cuda"), torch.zeros(1, N, device="cuda")
    err = WS._Err()
    check(lib.vl_nn_im2col(WS._p(x), 1, 1, 1, C, 1, kp, WS._p(cols), None))
    WS.gemm(cols, kp, w, kp, 1, N, kp, want, N, WS.EPI_BIAS, b, err)
    check(lib.vl_nn_conv_bf16(WS._p(x), 1, 1, 1, C, 1, 9, WS._p(w), kp, N, WS._p(got), N, WS._fp(b), WS.EPI_BIAS, err.ptr(), None))
    assert int(err.t.item()) == 0 and torch.equal(got, want) and float(want.abs().max()) > 0
