"""A convolution layer's gradients belong to the input of its forward pass, whatever becomes of that
tensor before the backward pass."""
import pytest

pytestmark = pytest.mark.gpu


def _layer(cin, cout, B, h, w, stride=1, seed=5):
    import torch
    from vortexlab_b200 import warmstart as WS
    c = WS.Conv(cin, cout, stride=stride, seed=seed)
    c.alloc(B, h, w)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(B, h, w, cin, generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn(c.rows, cout, generator=g, device="cuda")
    return WS, c, x, dy


def _gradients(c, x, dy, err, between=lambda: None):
    import torch
    dx = torch.zeros(c.B * c.h * c.wd, c.cin, device="cuda")
    c.forward(x, err)
    between()
    c.backward(dy, dx, False, err)
    return [t.clone() for t in (c.y, c.gw, c.gb, dx)]


# grids that 64-pixel blocks do not divide: a direct forward pass, a weight gradient through the im2col matrix
@pytest.mark.parametrize("cin,cout,h,w,stride", [(32, 32, 10, 22, 1), (64, 32, 6, 130, 1), (32, 64, 20, 44, 2), (96, 32, 7, 9, 1)])
def test_input_changed_before_backward_on_odd_grids(gpu, cin, cout, h, w, stride):
    import torch
    WS, c, x, dy = _layer(cin, cout, 2, h, w, stride)
    assert c.direct and not c.direct_w
    err = WS._Err()
    want = _gradients(c, x, dy, err)
    got = _gradients(c, x, dy, err, lambda: x.mul_(-2))
    assert int(err.t.item()) == 0
    for a, b in zip(want, got):
        assert torch.equal(a, b)


def test_network_on_an_odd_grid(gpu):
    """The network gathers those matrices in its backward pass (it leaves the layers' inputs alone): the
    gradients of layers that gather in forward."""
    import torch
    from vortexlab_b200 import warmstart as WS
    grads = []
    for plain in (False, True):
        net = WS.UNet(levels=3, c0=32, seed=2)
        net.alloc(2, 24, 40)
        if plain:
            for c in net.layers():
                c.forward = lambda x, err, held=False, f=c.forward: f(x, err)
        g = torch.Generator(device="cuda").manual_seed(9)
        x = torch.randn(2, 24, 40, WS.CIN, generator=g, device="cuda").to(torch.bfloat16)
        out = net.forward(x).clone()
        net.backward(torch.randn(2 * 24 * 40, net.cout, generator=g, device="cuda"))
        net.check_errors()
        grads.append([out] + [t.clone() for c in net.layers() for t in (c.gw, c.gb)])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cin,cout,h,w,stride", [(32, 32, 8, 64, 1), (4, 32, 9, 33, 1), (64, 64, 16, 64, 2)])
def test_inference_input_changed_before_backward(gpu, cin, cout, h, w, stride):
    """An inference tensor carries no version: the layer keeps its own copy."""
    import torch
    WS, c, x, dy = _layer(cin, cout, 2, h, w, stride)
    assert c.direct_w
    err = WS._Err()
    if cin == 4:
        c.backward = lambda dy, dx, acc, err, f=c.backward: f(dy, None, acc, err, need_dx=False)
    want = _gradients(c, x, dy, err)
    with torch.inference_mode():
        xi = x * 1
        got = _gradients(c, xi, dy, err, lambda: xi.mul_(-2))
    assert int(err.t.item()) == 0
    for a, b in zip(want, got):
        assert torch.equal(a, b)
