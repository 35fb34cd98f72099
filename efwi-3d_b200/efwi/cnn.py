"""Small 3-D CNN of the learned gradient preconditioner on the engine's BF16
tensor-core convolutions (efwi_conv3d_forward / efwi_conv3d_wgrad).

Four 3x3x3 convolutions with 16 channels (ReLU after the first three),
BF16 weights and activations, FP32 accumulation; inputs of fewer than 16
channels are zero-padded.  Activations are channels-last [D][H][W][16].  The
FP32 master weights are cast to BF16 at every forward pass, so any torch
optimizer trains them.  No reference counterpart.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import math

import torch
from torch.autograd import forward_ad

from ._lib import lib

C16 = 16


def _ptr(t):
    return t.data_ptr() if t is not None else None


def _stream(dev):
    return C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


def _on(dev):
    """The device as the current one (nothing to do where it is already)."""
    if torch.cuda.current_device() == dev.index:
        return contextlib.nullcontext()
    return torch.cuda.device(dev)


def conv3d_raw(x: torch.Tensor, wb: torch.Tensor, bias, relu: bool, out_f32: bool = False):
    """x [D,H,W,16] bf16, wb [27,16,16] bf16 -> [D,H,W,16] (bf16, or f32)."""
    assert x.dtype == torch.bfloat16 and x.is_contiguous() and x.shape[-1] == C16
    assert wb.dtype == torch.bfloat16 and wb.is_contiguous() and tuple(wb.shape) == (27, C16, C16)
    D, H, W = x.shape[:3]
    yb = None if out_f32 else torch.empty_like(x)
    yf = torch.empty(x.shape, device=x.device, dtype=torch.float32) if out_f32 else None
    b = bias.float().contiguous() if bias is not None else None
    with _on(x.device):
        rc = lib().efwi_conv3d_forward(_ptr(x), _ptr(wb), _ptr(b), D, H, W, int(relu), _ptr(yb),
                                       _ptr(yf), _stream(x.device))
    if rc:
        raise RuntimeError(f"efwi_conv3d_forward failed ({rc})")
    return yf if out_f32 else yb


CONV_FORMS = {"mma": 0, "tcgen05": 1, "tcgen05-tma": 2, "tcgen05-tma3": 3, "tcgen05-ws": 4,
              "tcgen05-ws3": 5}


def set_conv_kernel(form: str) -> None:
    """Kernel of every later forward / input-gradient convolution of this
    process: 'mma' (mma.sync m16n8k16), 'tcgen05' (tensor-memory accumulator,
    one MMA per tap for 128 voxels, tile staged by loads), 'tcgen05-tma'
    (z-marching, one MMA per (dy, dx) for the three dz, planes staged by bulk
    tensor copies; the default), 'tcgen05-tma3' (one MMA per tap, tiles staged
    by bulk tensor copies three stages deep), 'tcgen05-ws' /
    'tcgen05-ws3' (warp-specialised: one warp issues the copies and MMAs,
    four drain the accumulators, mbarriers between them; two / three
    stages)."""
    if form not in CONV_FORMS:
        raise ValueError(f"unknown convolution kernel form {form!r}")
    lib().efwi_conv3d_set_kernel(CONV_FORMS[form])


def set_wgrad_kernel(form: str) -> None:
    """'tcgen05' (eight taps per MMA, accumulators in tensor memory; the
    default) or 'mma' (mma.sync) for every later weight-gradient
    convolution."""
    if form not in ("tcgen05", "mma"):
        raise ValueError(f"unknown weight-gradient kernel form {form!r}")
    lib().efwi_conv3d_set_wgrad_kernel(1 if form == "tcgen05" else 0)


def conv3d_status(device=None) -> bool:
    """True when a tcgen05 convolution since the last call gave up waiting for
    its tensor cores (its outputs are then incomplete); clears the flag."""
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    flag = C.c_int(0)
    with torch.cuda.device(dev):
        rc = lib().efwi_conv3d_status(C.byref(flag), _stream(dev))
    if rc:
        raise RuntimeError(f"efwi_conv3d_status failed ({rc})")
    return bool(flag.value)


def conv3d_wgrad(x: torch.Tensor, dy: torch.Tensor, nparts: int = 592) -> torch.Tensor:
    """dW[t][co][ci] = sum_v dy[v][co] x[v + off_t][ci] (f32)."""
    D, H, W = x.shape[:3]
    partial = torch.empty(nparts * 27 * C16 * C16, device=x.device, dtype=torch.float32)
    dw = torch.empty(27, C16, C16, device=x.device, dtype=torch.float32)
    with _on(x.device):
        rc = lib().efwi_conv3d_wgrad(_ptr(x), _ptr(dy), D, H, W, _ptr(partial), nparts, _ptr(dw),
                                     _stream(x.device))
    if rc:
        raise RuntimeError(f"efwi_conv3d_wgrad failed ({rc})")
    return dw


def _dense(t: torch.Tensor, dtype) -> torch.Tensor:
    """t as the kernels read it: of `dtype`, contiguous, on a 16-byte boundary
    (what saved-tensor hooks hand back need not be)."""
    if t.dtype == dtype and t.is_contiguous() and not t.data_ptr() & 15:
        return t
    t = t.to(dtype).contiguous()
    return t.clone() if t.data_ptr() & 15 else t


def conv3d_backward(x: torch.Tensor, wb: torch.Tensor, gy: torch.Tensor, y, want_dx: bool,
                    nparts: int = 592):
    """(dx or None, dw, db) of one layer: g = gy * (y > 0) in float32 (y None:
    no ReLU), dx and dw from g in BF16, db = sum of g over the voxels.  A gy
    [D, H, W] is the gradient of channel 0 alone."""
    D, H, W = x.shape[:3]
    kind = 2 if gy.dim() == 3 else int(gy.dtype != torch.bfloat16)
    gy = _dense(gy, torch.float32 if kind else torch.bfloat16)
    relu = int(y is not None)
    L = lib()
    n = L.efwi_conv3d_backward_scratch(D, H, W, nparts, kind, relu)
    scratch = torch.empty(n, device=x.device, dtype=torch.uint8)
    dx = torch.empty_like(x) if want_dx else None
    dw = torch.empty(27, C16, C16, device=x.device, dtype=torch.float32)
    db = torch.empty(C16, device=x.device, dtype=torch.float32)
    with _on(x.device):
        rc = L.efwi_conv3d_backward(_ptr(x), _ptr(wb), _ptr(gy), kind, _ptr(y),
                                    int(relu and y.dtype == torch.float32), D, H, W, _ptr(scratch),
                                    nparts, _ptr(dx), _ptr(dw), _ptr(db), _stream(x.device))
    if rc:
        raise RuntimeError(f"efwi_conv3d_backward failed ({rc})")
    return dx, dw, db


class Conv3dBF16(torch.autograd.Function):
    """One layer: y = relu?(conv(x, w) + b) with BF16 operands."""

    @staticmethod
    def forward(ctx, x, w, b, relu, out_f32):
        wb = w.to(torch.bfloat16).contiguous()
        y = conv3d_raw(x, wb, b, relu, out_f32)
        ctx.save_for_backward(x, wb, y)
        ctx.relu = relu
        return y

    @staticmethod
    def backward(ctx, gy):
        x, wb, y = ctx.saved_tensors
        bf16 = torch.bfloat16
        dx, dw, db = conv3d_backward(
            _dense(x, bf16), _dense(wb, bf16), gy,
            _dense(y, bf16 if y.dtype == bf16 else torch.float32) if ctx.relu else None,
            ctx.needs_input_grad[0])
        if torch.is_grad_enabled():  # create_graph: db stays a function of gy
            g = gy.float()
            db = (g * (y > 0) if ctx.relu else g).sum(dim=(0, 1, 2))
        return dx, dw, db, None, None


class _Network(torch.autograd.Function):
    """The network's layers as one node: ReLU layers, then channel 0 of the
    last layer, [D, H, W] f32 (its other channels are neither written nor
    differentiated).  Same kernels and sums as a chain of Conv3dBF16; what
    it saves is the host work between their launches.  `keep`: a backward pass
    may follow; otherwise an activation lives until the next one is there."""

    @staticmethod
    def forward(ctx, x, n, keep, *params):
        ws, bs = params[:n], params[n:]
        if any(p.device != x.device for p in params):
            raise ValueError("the network's parameters and input are on different devices")
        wb = torch.stack([w.detach() for w in ws]).to(torch.bfloat16)
        assert tuple(wb.shape) == (n, 27, C16, C16)
        bias = [b.detach().float().contiguous() for b in bs]
        D, H, W = x.shape[:3]
        L, acts, h, rc = lib(), [], x, 0
        with _on(x.device):
            st = _stream(x.device)
            for k in range(n - 1):
                y = torch.empty_like(x)
                rc = rc or L.efwi_conv3d_forward(_ptr(h), _ptr(wb[k]), _ptr(bias[k]), D, H, W, 1,
                                                 _ptr(y), None, st)
                if keep:
                    acts.append(y)
                h = y
            out = torch.empty(D, H, W, device=x.device, dtype=torch.float32)
            head = rc or L.efwi_conv3d_forward_head(_ptr(h), _ptr(wb[n - 1]), _ptr(bias[n - 1]), D,
                                                    H, W, 0, _ptr(out), st)
        if rc or head not in (0, 3):
            raise RuntimeError(f"a convolution of the network failed ({rc or head})")
        if head == 3:  # another kernel form is selected
            out = conv3d_raw(h, wb[n - 1], bs[n - 1], False, True)[..., 0].contiguous()
        if keep:
            ctx.save_for_backward(x, wb, *acts)
        return out

    @staticmethod
    def backward(ctx, gy):
        x, wb, *acts = (_dense(t, torch.bfloat16) for t in ctx.saved_tensors)
        n = wb.shape[0]
        dws, dbs, g = [None] * n, [None] * n, gy
        for k in range(n - 1, -1, -1):
            g, dws[k], dbs[k] = conv3d_backward(acts[k - 1] if k else x, wb[k], g,
                                                acts[k] if k < n - 1 else None,
                                                k > 0 or ctx.needs_input_grad[0])
        if torch.is_grad_enabled():  # create_graph: the head's db stays a function of gy
            dbs[-1] = torch.nn.functional.pad(gy.float().sum().reshape(1), (0, C16 - 1))
        return (g, None, None, *dws, *dbs)


class _ChannelsLast(torch.autograd.Function):
    @staticmethod
    def forward(ctx, feats):
        ctx.c = feats.shape[0]
        f = feats.contiguous()
        x = torch.empty(feats.shape[1:] + (C16,), device=feats.device, dtype=torch.bfloat16)
        with _on(f.device):
            rc = lib().efwi_channels_last(_ptr(f), ctx.c, x.numel() // C16, _ptr(x),
                                          _stream(f.device))
        if rc:
            raise RuntimeError(f"efwi_channels_last failed ({rc})")
        return x

    @staticmethod
    def backward(ctx, gx):
        return gx[..., :ctx.c].permute(3, 0, 1, 2).to(torch.float32)


def _transformed(t: torch.Tensor) -> bool:
    """Whether t takes part in a functorch transform, forward-mode
    differentiation or a trace, which see torch operations only."""
    return (type(t) not in (torch.Tensor, torch.nn.Parameter)
            or torch._C._are_functorch_transforms_active()
            or forward_ad.unpack_dual(t).tangent is not None
            or torch.jit.is_tracing() or torch.compiler.is_compiling())


def to_channels_last(feats: torch.Tensor) -> torch.Tensor:
    """[C, D, H, W] f32 -> [D, H, W, 16] bf16 (channels zero-padded)."""
    c = feats.shape[0]
    if (feats.is_cuda and feats.dtype == torch.float32 and feats.dim() == 4 and 1 <= c <= C16
            and feats.numel() > 0 and not _transformed(feats)):
        return _ChannelsLast.apply(feats)
    x = torch.zeros(feats.shape[1:] + (C16,), device=feats.device, dtype=torch.bfloat16)
    x[..., :c] = feats.permute(1, 2, 3, 0).to(torch.bfloat16)
    return x


class Preconditioner(torch.nn.Module):
    """(gradient, model, illumination) -> update direction."""

    def __init__(self, cin: int = 3, seed: int = 0, layers: int = 4):
        super().__init__()
        gen = torch.Generator().manual_seed(seed)
        ws, bs = [], []
        for k in range(layers):
            fan_in = 27 * (cin if k == 0 else C16)
            w = torch.randn(27, C16, C16, generator=gen) * math.sqrt(2.0 / fan_in)
            if k == 0:
                w[:, :, cin:] = 0.0
            if k == layers - 1:
                w[:, 1:, :] = 0.0
                w *= 0.1
            ws.append(torch.nn.Parameter(w))
            bs.append(torch.nn.Parameter(torch.zeros(C16)))
        self.w = torch.nn.ParameterList(ws)
        self.b = torch.nn.ParameterList(bs)

    def forward(self, feats: torch.Tensor) -> torch.Tensor:
        """feats [C, D, H, W] f32 on a GPU -> [D, H, W] f32."""
        h = to_channels_last(feats)
        params = (*self.w, *self.b)
        if not params:
            return h[..., 0]
        keep = torch.is_grad_enabled() and (h.requires_grad or any(p.requires_grad for p in params))
        return _Network.apply(h, len(params) // 2, keep, *params)
