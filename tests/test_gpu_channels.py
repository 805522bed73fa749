"""The network's channel moves and the ReLU backward pass, in groups of 16 bytes and (where counts, offsets
or addresses do not allow it) one value at a time, against torch: whole results, equal bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,ctot,coff", [(32, 96, 64), (64, 64, 0), (8, 24, 8), (12, 20, 4), (5, 9, 3), (32, 40, 4)])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 3, 5), (1, 16, 33)])
def test_channel_moves(gpu, B, H, W, C, ctot, coff):
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(B, H, W, C, generator=g, device="cuda").to(torch.bfloat16)
    y = torch.full((B, 2 * H, 2 * W, ctot), 7.0, dtype=torch.bfloat16, device="cuda")
    want = y.clone()
    want[..., coff:coff + C] = x.repeat_interleave(2, 1).repeat_interleave(2, 2)
    check(lib.vl_nn_up2(WS._p(x), B, H, W, C, WS._p(y), ctot, coff, None))
    assert torch.equal(y, want)
    R = B * H * W
    y = torch.full((R, ctot), 7.0, dtype=torch.bfloat16, device="cuda")
    want = y.clone()
    want[:, coff:coff + C] = x.reshape(R, C)
    check(lib.vl_nn_copy_channels(WS._p(x), R, C, WS._p(y), ctot, coff, None))
    assert torch.equal(y, want)
    d = torch.randn(B, 2 * H, 2 * W, ctot, generator=g, device="cuda")
    for acc in (0, 1):
        o = torch.randn(4 * R, C, generator=g, device="cuda")
        part = d.reshape(4 * R, ctot)[:, coff:coff + C]
        want = o + part if acc else part.clone()
        check(lib.vl_nn_slice_channels(WS._p(d), 4 * R, ctot, coff, C, WS._p(o), acc, None))
        assert torch.equal(o, want)
        o = torch.randn(B, H, W, C, generator=g, device="cuda")
        q = d.reshape(B, H, 2, W, 2, ctot)[..., coff:coff + C]
        s = ((q[:, :, 0, :, 0] + q[:, :, 0, :, 1]) + q[:, :, 1, :, 0]) + q[:, :, 1, :, 1]
        want = o + s if acc else s
        check(lib.vl_nn_up2_bwd(WS._p(d), B, H, W, C, ctot, coff, WS._p(o), acc, None))
        assert torch.equal(o, want)


@pytest.mark.parametrize("R,C", [(1, 4), (31, 32), (257, 36), (1000, 8), (512, 128), (300, 5)])
@pytest.mark.parametrize("relu", [0, 1])
def test_relu_backward(gpu, R, C, relu):
    """dz and the 32-row column sums: the grouped kernel (no transposed copy asked for) against the one that
    also transposes; the bias gradient against FP64 (at most R terms, each rounded to BF16 first)."""
    import torch
    from vortexlab_b200 import warmstart as WS
    from vortexlab_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(4)
    dy = torch.randn(R, C, generator=g, device="cuda")
    y = torch.randn(R, C, generator=g, device="cuda").relu().to(torch.bfloat16)
    out = []
    for transposed in (False, True):
        dz = torch.full((R + 1, C), 7.0, dtype=torch.bfloat16, device="cuda")
        dzt = torch.zeros(C, R, dtype=torch.bfloat16, device="cuda")
        cs = torch.full((C, (R + 31) // 32), 7.0, device="cuda")
        db = torch.zeros(C, device="cuda")
        check(lib.vl_nn_act_bwd(WS._p(dy), WS._p(y) if relu else None, R, C, relu, WS._p(dz), WS._p(dzt) if transposed else None,
                                WS._p(cs), None))
        check(lib.vl_nn_bias_grad(WS._p(cs), R, C, WS._p(db), None))
        out.append((dz, cs, db))
    want = (dy * (y.float() > 0) if relu else dy).to(torch.bfloat16)
    for dz, cs, db in out:
        assert torch.equal(dz[:R], want) and bool((dz[R] == 7.0).all())
        exact = want.double().sum(0)
        assert bool(((db.double() - exact).abs() <= R * 2.0 ** -24 * want.double().abs().sum(0)).all())
    assert torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][2], out[1][2])
