"""The fused backward pass of a convolution layer against its parts: masked
gradient, input gradient and weight gradient the same bits, bias gradient
against float64; and the z-marching forward against the one-tap form at the
edges of its tiles and z ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 16, 8), (5, 17, 9), (2, 40, 31), (33, 5, 20)])
@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("out_f32", [True, False])
@pytest.mark.parametrize("want_dx", [True, False])
def test_backward_matches_its_parts(shape, relu, out_f32, want_dx):
    from efwi.cnn import conv3d_backward, conv3d_raw, conv3d_status, conv3d_wgrad
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(*shape, 16, device="cuda", generator=g).to(torch.bfloat16)
    wb = torch.randn(27, 16, 16, device="cuda", generator=g).to(torch.bfloat16)
    dt = torch.float32 if out_f32 else torch.bfloat16
    y = torch.randn(*shape, 16, device="cuda", generator=g).to(dt)
    gy = torch.randn(*shape, 16, device="cuda", generator=g).to(dt)
    gr = gy.float()
    if relu:
        gr = gr * (y > 0)
    dx, dw, db = conv3d_backward(x, wb, gy, y if relu else None, want_dx)
    dyb = gr.to(torch.bfloat16)
    wt = wb.flip(0).transpose(1, 2).contiguous()
    assert (dx is None) == (not want_dx)
    if want_dx:
        assert torch.equal(dx, conv3d_raw(dyb, wt, None, False))
    assert torch.equal(dw, conv3d_wgrad(x, dyb))
    # a float32 sum of n terms in a tree of partial sums: a few roundings each
    ref, size = gr.double().sum(dim=(0, 1, 2)), gr.double().abs().sum(dim=(0, 1, 2))
    assert bool(((db.double() - ref).abs() <= 32 * 2.0 ** -24 * size).all())
    assert not conv3d_status()


def test_backward_keeps_infinities_and_nans():
    """An infinite gradient behind a closed ReLU is NaN, as in gy * (y > 0)."""
    from efwi.cnn import conv3d_backward
    x = torch.ones(2, 2, 2, 16, device="cuda", dtype=torch.bfloat16)
    wb = torch.zeros(27, 16, 16, device="cuda", dtype=torch.bfloat16)
    gy = torch.zeros_like(x)
    y = torch.ones_like(x)
    gy[0, 0, 0, 3] = float("inf")
    gy[0, 0, 0, 4] = float("inf")
    y[0, 0, 0, 4] = -1.0
    _, _, db = conv3d_backward(x, wb, gy, y, False)
    ref = (gy.float() * (y > 0)).sum(dim=(0, 1, 2))
    assert torch.equal(torch.isnan(db), torch.isnan(ref)) and torch.isinf(db[3])
    assert torch.equal(db[:3], ref[:3])


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 17, 9), (40, 15, 8), (70, 33, 7), (1, 300, 200),
                                   (20, 300, 297)])
def test_z_march_matches_single_tap_form(shape):
    from efwi.cnn import conv3d_raw, conv3d_status, set_conv_kernel
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    x = torch.randn(*shape, 16, device="cuda", generator=g).to(torch.bfloat16)
    wb = torch.randn(27, 16, 16, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(16, device="cuda", generator=g)
    out = {}
    try:
        for form in ("tcgen05", "tcgen05-tma"):
            set_conv_kernel(form)
            out[form] = (conv3d_raw(x, wb, b, True), conv3d_raw(x, wb, None, False, True))
    finally:
        set_conv_kernel("tcgen05-tma")
    for u, v in zip(out["tcgen05"], out["tcgen05-tma"]):
        assert torch.equal(u, v)
    assert not conv3d_status()


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 17, 9), (20, 16, 8)])
@pytest.mark.parametrize("form", ["tcgen05-tma", "mma"])
def test_network_node_matches_chain_of_layers(shape, form):
    """One autograd node for the network, its channel-0 head and its input
    copy against Conv3dBF16 layer by layer: the same bits, gradients of the
    input and all parameters included."""
    from efwi.cnn import Conv3dBF16, Preconditioner, set_conv_kernel
    g = torch.Generator(device="cuda").manual_seed(7)
    feats = torch.randn(3, *shape, device="cuda", generator=g)
    gy = torch.randn(*shape, device="cuda", generator=g)
    net = Preconditioner(seed=3).cuda()
    with torch.no_grad():
        for p in net.b:
            p += 0.1
    try:
        set_conv_kernel(form)
        a = feats.clone().requires_grad_(True)
        ya = net(a)
        ga = torch.autograd.grad(ya, [a, *net.parameters()], gy)
        b = feats.clone().requires_grad_(True)
        h = torch.zeros(shape + (16,), device="cuda", dtype=torch.bfloat16)
        h[..., :3] = b.permute(1, 2, 3, 0).to(torch.bfloat16)
        n = len(net.w)
        for k in range(n):
            h = Conv3dBF16.apply(h, net.w[k], net.b[k], k < n - 1, k == n - 1)
        yb = h[..., 0]
        gb = torch.autograd.grad(yb, [b, *net.parameters()], gy)
    finally:
        set_conv_kernel("tcgen05-tma")
    assert torch.equal(ya, yb)
    for u, v in zip(ga, gb):
        assert torch.equal(u, v)
