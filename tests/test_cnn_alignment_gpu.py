"""Weights and outputs of a convolution on any boundary that their type allows:
the tensor-memory forms hand calls off 16 bytes to the mma.sync kernel."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _ready():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _at(n, offset, dtype=torch.bfloat16):
    """n elements `offset` elements off a 16-byte boundary."""
    buf = torch.empty(n + offset, device="cuda", dtype=dtype)
    return buf[offset:]


@pytest.mark.parametrize("off_w,off_y", [(0, 1), (1, 0), (1, 1), (2, 2), (3, 5), (8, 1)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 9, 17)])
def test_forward_at_any_element_boundary(off_w, off_y, shape):
    from efwi._lib import lib
    from efwi.cnn import conv3d_raw, set_conv_kernel
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(*shape, 16, device="cuda", generator=g).to(torch.bfloat16)
    wb = torch.randn(27, 16, 16, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(16, device="cuda", generator=g)
    try:
        set_conv_kernel("mma")
        ref = conv3d_raw(x, wb, b, True)
    finally:
        set_conv_kernel("tcgen05-tma")
    w = _at(wb.numel(), off_w).copy_(wb.reshape(-1))
    y = _at(x.numel(), off_y)
    D, H, W = shape
    rc = lib().efwi_conv3d_forward(x.data_ptr(), w.data_ptr(), b.data_ptr(), D, H, W, 1, y.data_ptr(),
                                   None, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert torch.equal(y.view(x.shape), ref)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_layer_with_weights_off_16_bytes(offset):
    """BF16 weights are used where they lie, forward and backward."""
    from efwi.cnn import Conv3dBF16, set_conv_kernel
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(3, 5, 9, 16, device="cuda", generator=g).to(torch.bfloat16).requires_grad_(True)
    w0 = torch.randn(27, 16, 16, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(16, device="cuda", generator=g)
    w1 = _at(w0.numel(), offset).copy_(w0.reshape(-1)).view(w0.shape)
    assert w1.data_ptr() & 15
    out = []
    try:
        set_conv_kernel("mma")
        for w in (w0, w1):
            y = Conv3dBF16.apply(x, w, b, True, False)
            out.append((y, torch.autograd.grad(y, x, torch.ones_like(y))[0]))
    finally:
        set_conv_kernel("tcgen05-tma")
    for u, v in zip(*out):
        assert torch.equal(u, v)
