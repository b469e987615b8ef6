"""Torch-tensor front ends of the C-ABI kernels that surround the attention in an MVPFormer block,
its encoder and its heads (``include/mvpa.h``: mvpa_rmsnorm, mvpa_silu_mul, mvpa_wave_encode,
mvpa_channel_mean, mvpa_contrastive_logits, and the backwards mvpa_rmsnorm_bwd, mvpa_silu_mul_bwd).
`rmsnorm_train` and `swiglu` are differentiable and take any tensor (torch expressions serve what the
kernels do not); the others are forward only, CUDA tensors, bf16 or fp32.
"""
from __future__ import annotations

import ctypes
import functools

import numpy as np
import torch

import mvpa_host as _host
import mvpa_native as _nat


def _code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _nat.MVPA_BF16
    if t.dtype == torch.float32:
        return _nat.MVPA_F32
    raise RuntimeError(f"mvpa_ops: dtype {t.dtype} not supported (bfloat16 or float32)")


def _stream(t: torch.Tensor) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("mvpa_ops: tensors must be on a CUDA device (no CPU path)")


def rmsnorm(x, weight, eps, add=None, sum_out=None, out=None):
    """y = rmsnorm(h) * weight over the last dimension, h = x (+ add).  With `add`, h is written to `sum_out`
    (which may be `x` itself: the update is elementwise).  Returns y."""
    _need_cuda(x, weight, add)
    E = x.shape[-1]
    x2 = x.reshape(-1, E)
    assert x2.is_contiguous() and weight.is_contiguous() and weight.dtype == x.dtype
    y = torch.empty_like(x2) if out is None else out
    if add is not None:
        assert add.dtype == x.dtype and add.reshape(-1, E).is_contiguous()
    with _nat.on_device(x.device):
        st = _nat.lib().mvpa_rmsnorm(x2.data_ptr(), add.data_ptr() if add is not None else None, weight.data_ptr(),
                                     sum_out.data_ptr() if sum_out is not None else None, y.data_ptr(), x2.shape[0], E,
                                     float(eps), _code(x), _stream(x))
    _nat.check(st, "mvpa_rmsnorm")
    return y.view(x.shape)


def silu_mul(gate, up, out):
    """out = silu(gate) * up for 2-D views with unit inner stride (column blocks of wider buffers are fine)."""
    _need_cuda(gate, up, out)
    rows, width = gate.shape
    assert up.shape == gate.shape and out.shape == gate.shape
    assert gate.stride(1) == up.stride(1) == out.stride(1) == 1 and gate.stride(0) == up.stride(0)
    with _nat.on_device(gate.device):
        st = _nat.lib().mvpa_silu_mul(gate.data_ptr(), up.data_ptr(), gate.stride(0), out.data_ptr(), out.stride(0), rows,
                                      width, _code(gate), _stream(gate))
    _nat.check(st, "mvpa_silu_mul")
    return out


def rmsnorm_bwd(x, weight, dy, eps, add=None):
    """Gradients (dx, dweight) of `rmsnorm(x, weight, eps)` (no residual) for the incoming gradient `dy`; `add`, the
    gradient that reaches x on another way (a residual connection), is added to dx."""
    _need_cuda(x, weight, dy, add)
    E = x.shape[-1]
    x2, dy2 = x.reshape(-1, E), dy.reshape(-1, E)
    assert x2.is_contiguous() and dy2.is_contiguous() and weight.is_contiguous()
    assert weight.dtype == x.dtype == dy.dtype and dy.shape == x.shape
    if add is not None:
        assert add.dtype == x.dtype and add.is_contiguous() and add.numel() == x.numel()
    dx, dw = torch.empty(x.shape, dtype=x.dtype, device=x.device), torch.empty_like(weight)
    lib = _nat.lib()
    with _nat.on_device(x.device):   # (the size depends on the device's multiprocessors)
        nbytes = lib.mvpa_rmsnorm_bwd_workspace_bytes(x2.shape[0], E)
        ws = torch.empty(nbytes, dtype=torch.uint8, device=x.device)
        st = lib.mvpa_rmsnorm_bwd(x2.data_ptr(), weight.data_ptr(), dy2.data_ptr(), add.data_ptr() if add is not None else None,
                                  dx.data_ptr(), dw.data_ptr(), x2.shape[0], E, float(eps), _code(x), ws.data_ptr(), nbytes,
                                  _stream(x))
    _nat.check(st, "mvpa_rmsnorm_bwd")
    return dx, dw


def silu_mul_bwd(gate, up, dout):
    """Gradients (dgate, dup) of silu(gate) * up for 2-D tensors with unit inner stride."""
    _need_cuda(gate, up, dout)
    rows, width = gate.shape
    assert up.shape == gate.shape and dout.shape == gate.shape and gate.dtype == up.dtype == dout.dtype
    assert gate.stride(1) == up.stride(1) == dout.stride(1) == 1 and gate.stride(0) == up.stride(0)
    dgate, dup = (torch.empty((rows, width), dtype=gate.dtype, device=gate.device) for _ in range(2))
    with _nat.on_device(gate.device):
        st = _nat.lib().mvpa_silu_mul_bwd(gate.data_ptr(), up.data_ptr(), gate.stride(0), dout.data_ptr(), dout.stride(0),
                                          dgate.data_ptr(), dup.data_ptr(), width, rows, width, _code(gate), _stream(gate))
    _nat.check(st, "mvpa_silu_mul_bwd")
    return dgate, dup


def _plain(*ts):
    """Tensors that the kernels can take and that nothing traces: ordinary CUDA tensors of one supported dtype,
    contiguous, 16-byte aligned, not empty; no forward-mode level, functorch transform or tracer is active
    (those are served by the differentiable torch expressions)."""
    t0 = ts[0]
    if _host.usable(t0):
        answer = _host.module().plain(*ts)
        if answer >= 0:
            return answer == 1
    # (a function mode is active, or the first tensor is none of ours; types first: a symbolic value answers no question about itself)
    if not all(type(t) in (torch.Tensor, torch.nn.Parameter) for t in ts) or not _nat.untraced() \
            or t0.dtype not in (torch.bfloat16, torch.float32):
        return False
    # (a backward may run on a thread of the autograd engine, where a transform shows on the tensor alone)
    if any(torch._C._functorch.is_functorch_wrapped_tensor(t) or not torch._C._has_storage(t) for t in ts):
        return False
    return all(t.is_cuda and t.dtype == t0.dtype and t.device == t0.device
               and t.is_contiguous() and t.numel() > 0 and t.data_ptr() % 16 == 0 for t in ts)


def _rows_fit(t):
    """The row kernels' widths: whole 16-byte vectors, at most 512 of them."""
    nbytes = t.shape[-1] * t.element_size() if t.dim() else 0
    return nbytes % 16 == 0 and nbytes <= 512 * 16


class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, eps):
        ctx.save_for_backward(x, weight)
        ctx.eps = eps
        y = torch.empty_like(x)          # (not a view of one: the caller may change it in place)
        rmsnorm(x, weight, eps, out=y)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        if not torch.is_grad_enabled() and _plain(x, weight, dy.contiguous()):
            return (*rmsnorm_bwd(x, weight, dy.contiguous(), ctx.eps), None)
        # a graph of the gradient is wanted (or a transform is active): the same formula in torch operations
        xf, wf, g = x.float(), weight.float(), dy.float()
        rstd = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + ctx.eps)
        xh, gw = xf * rstd, g * wf
        dx = rstd * (gw - xh * (gw * xh).mean(-1, keepdim=True))
        return dx.to(x.dtype), (g * xh).sum(dim=tuple(range(x.dim() - 1))).to(weight.dtype), None


def rmsnorm_train(x, weight, eps):
    """Differentiable `x * rsqrt(mean(x^2) + eps) * weight` over the last dimension, in fp32, rounded once: one
    kernel forward and two backward where the kernels apply, torch operations everywhere else."""
    if _plain(x, weight) and _rows_fit(x) and x.dim() > 0 and weight.shape == x.shape[-1:]:
        return _RMSNorm.apply(x, weight, eps)
    xf = x.float()
    return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * weight.float()).to(x.dtype)


class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate, up):
        ctx.save_for_backward(gate, up)
        w = gate.shape[-1]
        out = torch.empty_like(gate)     # (not a view of one, as above)
        silu_mul(gate.view(-1, w), up.view(-1, w), out.view(-1, w))
        return out

    @staticmethod
    def backward(ctx, dout):
        gate, up = ctx.saved_tensors
        if not torch.is_grad_enabled() and _plain(gate, up, dout.contiguous()):
            w = gate.shape[-1]
            dgate, dup = silu_mul_bwd(gate.view(-1, w), up.view(-1, w), dout.contiguous().view(-1, w))
            return dgate.view(gate.shape), dup.view(gate.shape)
        gf, d = gate.float(), dout.float()
        s = torch.sigmoid(gf)
        return (d * up.float() * (s * (1 + gf * (1 - s)))).to(gate.dtype), (d * (gf * s)).to(up.dtype)


def swiglu(gate, up):
    """Differentiable silu(gate) * up: one kernel each way where the kernels apply, torch operations elsewhere."""
    if _plain(gate, up) and gate.shape == up.shape and gate.dim() > 0 and gate.shape[-1] * gate.element_size() % 16 == 0:
        return _SwiGLU.apply(gate, up)
    return torch.nn.functional.silu(gate) * up


@functools.lru_cache(maxsize=None)
def db4_filters():
    """Decomposition filters (dec_lo, dec_hi) of the Daubechies wavelet with four vanishing moments, eight
    taps, derived numerically: |H(w)|^2 = 2 cos^8(w/2) P(sin^2(w/2)), P(y) = 1 + 4y + 10y^2 + 20y^3;
    the roots of P map to z through y = (2 - z - 1/z) / 4, the three roots inside the unit circle give the
    minimum-phase ("extremal phase") scaling filter h, normalised to sum sqrt(2).  Conventions of `pywt`
    (which `models/fftencoder.py:62` takes its filters from): dec_lo = h reversed, dec_hi[k] = -(-1)^k h[k]."""
    y_roots = np.roots([20.0, 10.0, 4.0, 1.0])
    z_roots = []
    for y in y_roots:
        pair = np.roots([1.0, -(2.0 - 4.0 * y), 1.0])
        z_roots.append(pair[np.argmin(np.abs(pair))])
    h = np.poly(np.concatenate([-np.ones(4), np.array(z_roots)])).real
    h *= np.sqrt(2.0) / h.sum()
    dec_lo = h[::-1].copy()
    dec_hi = np.array([-((-1) ** k) * h[k] for k in range(8)])
    return dec_lo.astype(np.float32), dec_hi.astype(np.float32)


def wave_sizes(segment_len: int):
    """(per-level coefficient counts finest first, total row length) of the encoder's transform."""
    levels = (ctypes.c_int32 * 16)()
    total = _nat.lib().mvpa_wave_encode_size(int(segment_len), levels, 16)
    sizes, n = [], segment_len
    while len(sizes) < 16 and levels[len(sizes)] > 0:
        sizes.append(int(levels[len(sizes)]))
    return sizes, int(total)


def wave_encode(x, ln_weight, eps=1e-5, pad_to=None):
    """x (rows, len) fp32 / bf16 -> (rows, pad_to or total) in ln_weight's dtype: wavelet coefficients of every
    level, RMS-normalised and scaled by ln_weight; columns past the coefficient count are zero."""
    _need_cuda(x, ln_weight)
    rows, n = x.shape
    assert x.stride(1) == 1
    _, total = wave_sizes(n)
    ld_out = total if pad_to is None else int(pad_to)
    assert ln_weight.numel() == total and ln_weight.is_contiguous()
    out = torch.empty((rows, ld_out), dtype=ln_weight.dtype, device=x.device)
    lo, hi = db4_filters()
    fp = ctypes.POINTER(ctypes.c_float)
    with _nat.on_device(x.device):
        st = _nat.lib().mvpa_wave_encode(x.data_ptr(), x.stride(0), _code(x), lo.ctypes.data_as(fp), hi.ctypes.data_as(fp),
                                         ln_weight.data_ptr(), out.data_ptr(), ld_out, _code(ln_weight), rows, n,
                                         float(eps), _stream(x))
    _nat.check(st, "mvpa_wave_encode")
    return out


def channel_mean(h):
    """h (B,T,C,E) -> (B,E): mean over the channels of the last time step."""
    _need_cuda(h)
    B, T, C, E = h.shape
    assert h.is_contiguous()
    out = torch.empty((B, E), dtype=h.dtype, device=h.device)
    with _nat.on_device(h.device):
        st = _nat.lib().mvpa_channel_mean(h.data_ptr(), out.data_ptr(), B, T, C, E, _code(h), _stream(h))
    _nat.check(st, "mvpa_channel_mean")
    return out


def contrastive_logits(pred, enc, negatives, temperature):
    """pred, enc (B,T,C,E); negatives (B,T,C,K) int32 rows of enc.view(-1, E).  Returns (B*(T-1)*C, 1+K) fp32."""
    _need_cuda(pred, enc, negatives)
    B, T, C, E = pred.shape
    K = negatives.shape[-1]
    assert enc.shape == pred.shape and pred.is_contiguous() and enc.is_contiguous() and enc.dtype == pred.dtype
    assert negatives.dtype == torch.int32 and negatives.is_contiguous() and negatives.shape[:3] == (B, T, C)
    out = torch.empty((B * (T - 1) * C, K + 1), dtype=torch.float32, device=pred.device)
    with _nat.on_device(pred.device):
        st = _nat.lib().mvpa_contrastive_logits(pred.data_ptr(), enc.data_ptr(), negatives.data_ptr(), out.data_ptr(), B, T,
                                                C, E, K, float(temperature), _code(pred), _stream(pred))
    _nat.check(st, "mvpa_contrastive_logits")
    return out
