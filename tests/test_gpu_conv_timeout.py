"""A load that never arrives: every wait of the convolution kernels is bounded, the error flag is set, and the next
call is right (the tensor memory was given back)."""
import pytest

pytestmark = pytest.mark.gpu


def _data(B, H, W, C, N, stride):
    import torch
    from vortexlab_b200 import warmstart as WS
    g = torch.Generator(device="cuda").manual_seed(3)
    kp = WS._kp(9 * C)
    ho, wo = (H + stride - 1) // stride, (W + stride - 1) // stride
    x = torch.randn(B, H, W, C, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.zeros(N, kp, device="cuda")
    w[:, :9 * C] = 0.05 * torch.randn(N, 9 * C, generator=g, device="cuda")
    dz = torch.randn(B * ho * wo, N, generator=g, device="cuda").to(torch.bfloat16)
    return WS, kp, ho, wo, x, w.to(torch.bfloat16), dz


def _failed_then_right(WS, call, failing, out):
    import torch
    from vortexlab_b200._lib import check
    err = WS._Err()
    check(call(err))
    want = out.clone()
    assert int(err.t.item()) == 0
    for _ in range(3):
        check(failing(err))
    torch.cuda.synchronize()
    assert int(err.t.item()) == 1
    err = WS._Err()
    out.fill_(7.0)
    check(call(err))
    assert int(err.t.item()) == 0 and torch.equal(out, want)


# k_conv (64- and 32-channel chunks, stride 2, a K split), k_conv_rows, k_conv_first
@pytest.mark.parametrize("B,H,W,C,N,stride", [(2, 10, 22, 64, 32, 1), (2, 17, 51, 32, 64, 2), (1, 8, 16, 256, 256, 1), (4, 64, 256, 32, 32, 1),
                                              (8, 128, 256, 64, 64, 1), (4, 64, 128, 4, 32, 1)])
def test_convolution(gpu, B, H, W, C, N, stride):
    import torch
    from vortexlab_b200._lib import lib
    WS, kp, ho, wo, x, w, _ = _data(B, H, W, C, N, stride)
    out = torch.full((B * ho * wo, N), 7.0, device="cuda")
    call = lambda err, f=0: lib.vl_nn_conv_bf16(  # noqa: E731
        WS._p(x), B, H, W, C, stride, 9, WS._p(w), kp, N, WS._p(out), N, None, f, err.ptr(), None)
    _failed_then_right(WS, call, lambda err: call(err, 64), out)


# k_wgrad (both chunk widths, stride 2), k_wgrad_rows, k_wgrad_first
@pytest.mark.parametrize("B,H,W,C,N,stride", [(2, 8, 64, 64, 64, 1), (1, 16, 32, 32, 64, 1), (2, 16, 128, 64, 32, 2), (4, 64, 128, 32, 32, 1),
                                              (2, 32, 64, 192, 64, 1), (4, 64, 128, 4, 32, 1)])
def test_weight_gradient(gpu, B, H, W, C, N, stride):
    import torch
    from vortexlab_b200._lib import lib
    WS, kp, ho, wo, x, _, dz = _data(B, H, W, C, N, stride)
    gw = torch.full((kp, N), 7.0, device="cuda")
    args = lambda err: (WS._p(x), B, H, W, C, stride, WS._p(dz), N, WS._p(gw), kp, err.ptr(), None)  # noqa: E731
    _failed_then_right(WS, lambda err: lib.vl_nn_wgrad_bf16(*args(err)), lambda err: lib.vl_nn_wgrad_test_timeout(*args(err)), gw)


@pytest.mark.parametrize("B,H,W,C,N", [(2, 32, 64, 32, 64), (1, 15, 33, 64, 96), (1, 9, 17, 192, 64)])
def test_stride2_input_gradient(gpu, B, H, W, C, N):
    import torch
    from vortexlab_b200._lib import lib
    WS, kp, ho, wo, _, w, dz = _data(B, H, W, C, N, 2)
    wt = w.t().contiguous()
    dx = torch.full((B * H * W, C), 7.0, device="cuda")
    args = lambda err: (WS._p(dz), B, H, W, C, N, WS._p(wt), WS._p(dx), 0, err.ptr(), None)  # noqa: E731
    _failed_then_right(WS, lambda err: lib.vl_nn_dgrad2_bf16(*args(err)), lambda err: lib.vl_nn_dgrad2_test_timeout(*args(err)), dx)
