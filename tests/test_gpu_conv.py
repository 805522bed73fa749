"""The implicit convolution kernels (vl_nn_conv_bf16, vl_nn_wgrad_bf16) against the same products over the
materialised im2col matrix (vl_nn_im2col + vl_nn_gemm_bf16, tested against FP64 elsewhere): the K order and
the K splits are the same, so every result must be equal bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def _setup(B, H, W, C, stride, N, seed=1):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(B, H, W, C, generator=g, device="cuda").relu().to(torch.bfloat16)
    kp = WS._kp(9 * C)
    w = torch.zeros(N, kp, device="cuda")
    w[:, :9 * C] = 0.05 * torch.randn(N, 9 * C, generator=g, device="cuda")
    ho, wo = (H + stride - 1) // stride, (W + stride - 1) // stride
    cols = torch.zeros(B * ho * wo, kp, dtype=torch.bfloat16, device="cuda")
    check(lib.vl_nn_im2col(WS._p(x), B, H, W, C, stride, kp, WS._p(cols), None))
    return g, x, w.to(torch.bfloat16), cols, kp, ho, wo


# tile shapes 128 x 1 .. 8 x 16 and ragged rows of each, channel chunks of 32 and 64, one to several output
# channel blocks, both strides, K splits (FP32 results of few tiles), more tiles than blocks
@pytest.mark.parametrize("B,H,W,C,stride,N", [
    (1, 16, 32, 64, 1, 64), (1, 1, 1, 32, 1, 8), (2, 16, 64, 96, 1, 32), (1, 8, 128, 64, 1, 128), (2, 10, 22, 64, 1, 32),
    (3, 37, 53, 32, 1, 64), (1, 16, 64, 64, 2, 128), (2, 17, 51, 32, 2, 64), (1, 8, 16, 256, 1, 256), (1, 8, 16, 128, 1, 384),
    (1, 5, 130, 192, 1, 40), (2, 24, 144, 128, 2, 96), (16, 96, 130, 32, 1, 32), (4, 64, 256, 96, 1, 32),
    # the 4-channel input layer: a pixel, ragged tiles, more tiles than blocks
    (1, 1, 1, 4, 1, 8), (2, 7, 19, 4, 1, 32), (3, 33, 65, 4, 1, 72), (16, 96, 130, 4, 1, 32), (1, 4, 32, 4, 1, 256)])
@pytest.mark.parametrize("form", ["relu", "f32"])
def test_convolution(gpu, B, H, W, C, stride, N, form):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g, x, w, cols, kp, ho, wo = _setup(B, H, W, C, stride, N)
    R = B * ho * wo
    bias = torch.randn(N, generator=g, device="cuda")
    flags = WS.EPI_BIAS | WS.EPI_RELU | WS.EPI_BF16 if form == "relu" else 0
    dt = torch.bfloat16 if form == "relu" else torch.float32
    want = torch.full((R, N), 7.0, dtype=dt, device="cuda")
    got = torch.full((R + 1, N), 7.0, dtype=dt, device="cuda")      # one row more: nothing is written past the end
    err = WS._Err()
    WS.gemm(cols, kp, w, kp, R, N, kp, want, N, flags, bias, err)
    check(lib.vl_nn_conv_bf16(WS._p(x), B, H, W, C, stride, 9, WS._p(w), kp, N, WS._p(got), N,
                              WS._fp(bias) if form == "relu" else None, flags, err.ptr(), None))
    assert int(err.t.item()) == 0
    assert torch.equal(got[:R], want) and bool((got[R] == 7.0).all())


def test_convolution_accumulates_and_1x1(gpu):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    B, H, W, C, N = 2, 9, 33, 64, 64
    g, x, w, cols, kp, ho, wo = _setup(B, H, W, C, 1, N)
    R = B * H * W
    err = WS._Err()
    base = torch.randn(R, N, generator=g, device="cuda")
    one = torch.zeros(R, N, device="cuda")
    check(lib.vl_nn_conv_bf16(WS._p(x), B, H, W, C, 1, 9, WS._p(w), kp, N, WS._p(one), N, None, WS.EPI_BIAS * 0, err.ptr(), None))
    got = base.clone()
    check(lib.vl_nn_conv_bf16(WS._p(x), B, H, W, C, 1, 9, WS._p(w), kp, N, WS._p(got), N, None, WS.EPI_ACCUM, err.ptr(), None))
    # the K split of a product of few tiles is only taken without accumulation: equal to FP32 rounding
    assert torch.allclose(got, base + one, rtol=0, atol=2.0 ** -19 * float((base.abs() + one.abs()).max()))
    w1 = (0.1 * torch.randn(8, C, generator=g, device="cuda")).to(torch.bfloat16)
    b1 = torch.randn(8, generator=g, device="cuda")
    want = torch.zeros(R, 8, device="cuda")
    got = torch.zeros(R, 8, device="cuda")
    WS.gemm(x, C, w1, C, R, 8, C, want, 8, WS.EPI_BIAS, b1, err)
    check(lib.vl_nn_conv_bf16(WS._p(x), B, H, W, C, 1, 1, WS._p(w1), C, 8, WS._p(got), 8, WS._fp(b1), WS.EPI_BIAS, err.ptr(), None))
    assert int(err.t.item()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("B,H,W,C,stride,N", [
    (1, 16, 32, 64, 1, 64), (1, 16, 32, 32, 1, 32), (2, 16, 64, 96, 1, 32), (1, 8, 128, 64, 1, 128), (1, 16, 64, 64, 2, 128),
    (1, 8, 16, 256, 1, 256), (1, 8, 16, 128, 1, 384), (3, 64, 1, 32, 1, 8), (2, 30, 192, 160, 1, 72), (2, 33, 127, 96, 2, 64),
    (2, 128, 256, 192, 1, 64), (1, 1, 1, 4, 1, 8), (2, 7, 19, 4, 1, 32), (3, 33, 65, 4, 1, 72), (16, 96, 130, 4, 1, 32), (1, 4, 32, 4, 1, 256)])
def test_weight_gradient(gpu, B, H, W, C, stride, N):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g, x, _, cols, kp, ho, wo = _setup(B, H, W, C, stride, N)
    R = B * ho * wo
    if C > 4 and wo % 64 and (64 % wo or ho % (64 // wo)):
        pytest.skip("not a grid of whole 64-pixel blocks")
    dz = torch.randn(R, N, generator=g, device="cuda").to(torch.bfloat16)
    want = torch.full((kp, N), 7.0, device="cuda")
    got = torch.full((kp + 1, N), 7.0, device="cuda")
    err = WS._Err()
    WS.gemm(cols, kp, dz, N, kp, N, R, want, N, WS.A_MN | WS.B_MN, None, err)
    check(lib.vl_nn_wgrad_bf16(WS._p(x), B, H, W, C, stride, WS._p(dz), N, WS._p(got), kp, err.ptr(), None))
    assert int(err.t.item()) == 0
    assert torch.equal(got[:kp], want) and bool((got[kp] == 7.0).all())


@pytest.mark.parametrize("B,H,W,C,N", [(1, 16, 32, 32, 64), (2, 15, 33, 32, 32), (1, 1, 1, 8, 32), (1, 2, 3, 40, 96),
                                       (2, 32, 64, 128, 256), (3, 22, 70, 64, 128), (1, 9, 17, 192, 64), (4, 64, 256, 32, 64)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_stride2_input_gradient(gpu, B, H, W, C, N, accumulate):
    """Against dz W^T written out and gathered by col2im."""
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g, _, w, _, kp, ho, wo = _setup(B, H, W, C, 2, N)
    R = B * ho * wo
    dz = torch.randn(R, N, generator=g, device="cuda").to(torch.bfloat16)
    wt = w.t().contiguous()
    err = WS._Err()
    dcols = torch.zeros(R, kp, device="cuda")
    WS.gemm(dz, N, wt, N, R, kp, N, dcols, kp, 0, None, err)
    want = torch.randn(B * H * W + 1, C, generator=g, device="cuda")
    got = want.clone()
    check(lib.vl_nn_col2im(WS._p(dcols), B, H, W, C, 2, kp, WS._p(want), accumulate, None))
    check(lib.vl_nn_dgrad2_bf16(WS._p(dz), B, H, W, C, N, WS._p(wt), WS._p(got), accumulate, err.ptr(), None))
    assert int(err.t.item()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("stride,offset", [(1, 1), (1, 4), (2, 4), (2, 8)])
def test_layer_takes_input_gradients_at_any_alignment(gpu, stride, offset):
    """An input gradient that does not start on 32 bytes goes through the matrix, with the same values."""
    import torch
    from vortexlab_b200 import warmstart as WS
    g = torch.Generator(device="cuda").manual_seed(offset)
    B, H, W, C, N = 2, 16, 32, 32, 64
    c = WS.Conv(C, N, stride=stride, seed=3)
    c.alloc(B, H, W)
    err = WS._Err()
    x = torch.relu(torch.randn(B, H, W, C, generator=g, device="cuda")).bfloat16()
    dy = torch.randn(c.rows, N, generator=g, device="cuda")
    want = torch.zeros(B * H * W * C, device="cuda")
    got = torch.zeros(want.numel() + 32, device="cuda")[offset:offset + want.numel()]
    for dx in (want, got):
        c.forward(x, err)
        c.backward(dy, dx, False, err)
    assert int(err.t.item()) == 0 and torch.equal(got, want)


def test_input_changed_before_backward_is_refused(gpu):
    """The weight gradient reads the layer's input again."""
    import torch
    from vortexlab_b200 import warmstart as WS
    c = WS.Conv(32, 32, seed=3)
    c.alloc(1, 8, 64)
    x = torch.zeros(1, 8, 64, 32, dtype=torch.bfloat16, device="cuda")
    c.forward(x, None)
    x += 1
    with pytest.raises(RuntimeError, match="changed in place"):
        c.backward(torch.zeros(c.rows, 32, device="cuda"), None, False, None, need_dx=False)


def test_bad_arguments_are_refused(gpu):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import lib
    x = torch.zeros(1, 8, 8, 64, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(64, 576, dtype=torch.bfloat16, device="cuda")
    y = torch.zeros(64, 64, device="cuda")
    conv = lambda C=64, st=1, taps=9, kp=576, N=64, out=y: lib.vl_nn_conv_bf16(  # noqa: E731
        WS._p(x), 1, 8, 8, C, st, taps, WS._p(w), kp, N, WS._p(out), 64, None, 0, None, None)
    assert conv() == 0
    for bad in (dict(C=48), dict(st=3), dict(taps=4), dict(kp=512), dict(N=12), dict(out=y.reshape(-1)[4:])):
        assert conv(**bad) < 0, bad
    assert lib.vl_nn_wgrad_bf16(WS._p(x), 1, 8, 8, 48, 1, WS._p(w), 64, WS._p(y), 576, None, None) < 0
    assert lib.vl_nn_wgrad_bf16(WS._p(x), 1, 7, 9, 64, 1, WS._p(w), 64, WS._p(y), 576, None, None) < 0
