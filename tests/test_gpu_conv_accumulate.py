"""vl_nn_conv_bf16 with accumulation against im2col and the accumulating GEMM, which splits K where the tiles are few
whether it accumulates or not: the same sums, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


# no split (few K blocks; many tiles); a split of 64- and 32-channel chunks; a wider pitch; 1x1 with a split
@pytest.mark.parametrize("B,H,W,C,N,taps,pitch", [
    (2, 9, 33, 32, 64, 9, 64), (16, 64, 128, 128, 64, 9, 64), (1, 16, 32, 128, 64, 9, 64), (2, 10, 22, 96, 32, 9, 32),
    (1, 8, 16, 256, 256, 9, 264), (1, 7, 130, 192, 40, 9, 48), (1, 8, 16, 1024, 64, 1, 64)])
def test_accumulation(gpu, B, H, W, C, N, taps, pitch):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(B, H, W, C, generator=g, device="cuda").to(torch.bfloat16)
    kp = WS._kp(9 * C) if taps == 9 else C
    w = torch.zeros(N, kp, device="cuda")
    w[:, :taps * C] = 0.05 * torch.randn(N, taps * C, generator=g, device="cuda")
    w = w.to(torch.bfloat16)
    R = B * H * W
    cols = x.reshape(R, C)
    if taps == 9:
        cols = torch.zeros(R, kp, dtype=torch.bfloat16, device="cuda")
        check(lib.vl_nn_im2col(WS._p(x), B, H, W, C, 1, kp, WS._p(cols), None))
    want = torch.randn(R, pitch, generator=g, device="cuda")
    got = want.clone()
    err = WS._Err()
    for _ in range(2):
        WS.gemm(cols, kp, w, kp, R, N, kp, want, pitch, WS.EPI_ACCUM, None, err)
        check(lib.vl_nn_conv_bf16(WS._p(x), B, H, W, C, 1, taps, WS._p(w), kp, N, WS._p(got), pitch, None, WS.EPI_ACCUM,
                                  err.ptr(), None))
    assert int(err.t.item()) == 0 and torch.equal(got, want)
