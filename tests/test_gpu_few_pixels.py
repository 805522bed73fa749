"""The input gradient of a layer with few pixels and many output channels goes through the im2col matrix, whose GEMM is
split over the chip (the direct kernel had one block with a chain of 144 K steps): the bits of the direct kernel."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,B,h,w,matrix", [
    (64, 1024, 1, 8, 16, True), (64, 384, 1, 8, 16, True), (128, 512, 2, 10, 22, True), (256, 640, 1, 16, 32, True), (32, 512, 1, 32, 32, True),
    (64, 320, 1, 8, 16, False), (128, 384, 1, 8, 16, False), (256, 512, 1, 8, 16, False), (512, 640, 1, 16, 32, False),
    (64, 512, 1, 33, 32, False)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_input_gradient(gpu, cin, cout, B, h, w, matrix, accumulate):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    c = WS.Conv(cin, cout, seed=4)
    c.alloc(B, h, w)
    assert c.direct_x != matrix
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(B, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(c.rows, cout, generator=g, device="cuda")
    got = torch.randn(B * h * w, cin, generator=g, device="cuda")
    want = got.clone()
    err = WS._Err()
    c.forward(x, err)
    c.backward(dy, got, accumulate, err)
    check(lib.vl_nn_conv_bf16(WS._p(c.dz), B, h, w, cout, 1, 9, WS._p(c.wf), c.kpf, cin, WS._p(want), cin, None,
                              WS.EPI_ACCUM if accumulate else 0, err.ptr(), None))
    assert int(err.t.item()) == 0 and torch.equal(got, want)
