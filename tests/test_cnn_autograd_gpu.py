"""Autograd features around the preconditioner's convolutions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _layer(shape, seed=5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(*shape, 16, device="cuda", generator=g).to(torch.bfloat16)
    w = 0.2 * torch.randn(27, 16, 16, device="cuda", generator=g)
    b = torch.randn(16, device="cuda", generator=g)
    gy = torch.randn(*shape, 16, device="cuda", generator=g)
    return [t.requires_grad_(True) for t in (x, w, b)], gy


def _shift(t):  # on a 2- or 4-byte boundary
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    return buf[1:].view(t.shape)


HOOKS = {
    "permuted": (lambda t: t.transpose(0, 1).contiguous(), lambda t: t.transpose(0, 1)),
    "unaligned": (lambda t: t, _shift),
    "float64": (lambda t: t.double(), lambda t: t),
}


@pytest.mark.parametrize("hook", sorted(HOOKS))
@pytest.mark.parametrize("relu,out_f32", [(True, False), (True, True), (False, False)])
def test_layer_backward_under_saved_tensor_hooks(hook, relu, out_f32):
    """Whatever strides, alignment and type the hooks hand back."""
    from efwi.cnn import Conv3dBF16
    (x, w, b), gy = _layer((5, 7, 9))
    out = []
    for pack, unpack in ((lambda t: t, lambda t: t), HOOKS[hook]):
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            y = Conv3dBF16.apply(x, w, b, relu, out_f32)
        out.append(torch.autograd.grad(y, [x, w, b], gy.to(y.dtype)))
    for u, v in zip(*out):
        assert torch.equal(u, v)


@pytest.mark.parametrize("hook", sorted(HOOKS))
def test_network_backward_under_saved_tensor_hooks(hook):
    from efwi.cnn import Preconditioner
    net = Preconditioner(seed=2).cuda()
    feats = torch.randn(3, 5, 7, 9, device="cuda")
    out = []
    for pack, unpack in ((lambda t: t, lambda t: t), HOOKS[hook]):
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            y = net(feats)
        out.append(torch.autograd.grad(y, list(net.parameters()), torch.ones_like(y)))
    for u, v in zip(*out):
        assert torch.equal(u, v)


def _chain(feats):  # torch operations
    x = torch.zeros(feats.shape[1:] + (16,), device=feats.device, dtype=torch.bfloat16)
    x[..., :feats.shape[0]] = feats.permute(1, 2, 3, 0).to(torch.bfloat16)
    return x


def _dual(fn, a, t):
    from torch.autograd import forward_ad
    with forward_ad.dual_level():
        return forward_ad.unpack_dual(fn(forward_ad.make_dual(a, t))).tangent


TRANSFORMS = {
    "values": lambda fn, a, t: fn(a),
    "backward": lambda fn, a, t: torch.autograd.grad(fn(a.requires_grad_(True)).float().pow(2).sum(), a)[0],
    "grad": lambda fn, a, t: torch.func.grad(lambda v: fn(v).float().pow(2).sum())(a),
    "jvp": lambda fn, a, t: torch.func.jvp(fn, (a,), (t,))[1],
    "forward mode": _dual,
    "jacfwd": lambda fn, a, t: torch.func.jacfwd(lambda v: fn(v).float())(a),
    "jacrev": lambda fn, a, t: torch.func.jacrev(lambda v: fn(v).float())(a),
    "hvp": lambda fn, a, t: torch.autograd.functional.hvp(lambda v: fn(v).float().pow(3).sum(), a, t)[1],
    "trace": lambda fn, a, t: torch.jit.trace(fn, (a + 1,))(a),
}


@pytest.mark.parametrize("how", sorted(TRANSFORMS))
@pytest.mark.filterwarnings("ignore")
def test_channels_last_copy_under_transforms(how):
    from efwi.cnn import to_channels_last
    g = torch.Generator(device="cuda").manual_seed(1)
    a, t = (torch.randn(3, 2, 4, 5, device="cuda", generator=g) for _ in range(2))
    fn = TRANSFORMS[how]
    out, ref = fn(to_channels_last, a.clone(), t), fn(_chain, a.clone(), t)
    assert out.dtype == ref.dtype and torch.equal(out, ref)
    assert float(ref.abs().max()) > 0


@pytest.mark.parametrize("frozen", [True, False])
def test_inference_memory_does_not_grow_with_the_layers(frozen):
    """Without a backward pass to come (no_grad, or nothing to differentiate)
    the input copy and two activations of 2 * 16 bytes a voxel are alive."""
    from efwi.cnn import Preconditioner
    shape = (64, 64, 64)
    feats = torch.randn(3, *shape, device="cuda")
    unit = 32 * 64 ** 3
    for layers in (4, 12):
        net = Preconditioner(seed=2, layers=layers).cuda().requires_grad_(not frozen)
        with torch.set_grad_enabled(frozen):
            net(feats)
            torch.cuda.synchronize()
            base = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            y = net(feats)
            torch.cuda.synchronize()
        assert not y.requires_grad
        # and the output, a float a voxel, and the weights' BF16 copies
        assert torch.cuda.max_memory_allocated() - base <= 3 * unit + unit // 8 + (1 << 20)
        del y


@pytest.mark.parametrize("relu", [True, False])
def test_bias_gradient_can_be_differentiated_again(relu):
    """d/db sum_v (y_v)^2 = 2 sum_v m_v y_v (m: behind the ReLU), and again:
    2 times the number of open voxels.  Whole numbers in float32."""
    from efwi.cnn import Conv3dBF16
    (x, w, b), _ = _layer((5, 7, 9))
    y = Conv3dBF16.apply(x, w, b, relu, True)
    (db,) = torch.autograd.grad(y.pow(2).sum(), b, create_graph=True)
    ref = 2 * y.detach().double().sum(dim=(0, 1, 2))
    # sums of 315 terms in any order, each product rounded once
    size = 2 * y.detach().double().abs().sum(dim=(0, 1, 2))
    assert bool(((db.double() - ref).abs() <= 316 * 2.0 ** -24 * size).all())
    (d2,) = torch.autograd.grad(db.sum(), b)
    opened = (y > 0).sum(dim=(0, 1, 2)) if relu else torch.full((16,), 5 * 7 * 9, device="cuda")
    assert torch.equal(d2, 2.0 * opened)


def test_head_bias_gradient_can_be_differentiated_again():
    from efwi.cnn import Preconditioner
    net = Preconditioner(seed=2).cuda()
    y = net(torch.randn(3, 5, 7, 9, device="cuda"))
    b = net.b[-1]
    (db,) = torch.autograd.grad(y.pow(2).sum(), b, create_graph=True)
    (d2,) = torch.autograd.grad(db.sum(), b)
    assert torch.equal(d2, torch.tensor([630.0] + 15 * [0.0], device="cuda"))
