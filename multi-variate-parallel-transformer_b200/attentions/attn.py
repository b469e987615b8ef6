"""`flash_mvpa` — drop-in for the reference operator of the same name
(`attentions/attn.py:1317-1366`), backed by the sm_100a CUDA library.

Same signature and argument meaning as the reference.  What differs inside:
the relative-score matrices of `_rel_bias` (`attentions/attn.py:1305-1314`) are
never materialised, the Triton kernels are replaced by the C-ABI calls
`mvpa_fwd` / `mvpa_bwd` (``include/mvpa.h``), and the backward returns the
gradients of all eight tensors directly instead of leaving part of the work to
autograd.  There is no CPU path: tensors must live on a CUDA device.
"""
from __future__ import annotations

import ctypes
import math
import os
from operator import is_

import torch

import mvpa_host as _host
import mvpa_native as _nat


# MVPA_CHECK_STATUS=1: read the kernels' status word back after every forward and backward (synchronises).
_CHECK_STATUS = os.environ.get("MVPA_CHECK_STATUS", "0") == "1"


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _nat.MVPA_BF16
    if t.dtype == torch.float32:
        return _nat.MVPA_F32
    if t.dtype == torch.float16:
        return _nat.MVPA_F16
    raise RuntimeError(f"flash_mvpa: dtype {t.dtype} not supported (bfloat16, float16 or float32)")


def _tensor(t: torch.Tensor) -> _nat.Tensor:
    strides = t.stride()
    return _nat.Tensor(t.data_ptr(), strides[0], strides[1], strides[2])


def _aligned(t: torch.Tensor) -> bool:
    """A contiguous last dimension, 16-byte aligned base and strides: what the kernels read in place."""
    strides = t.stride()
    return strides[-1] == 1 and not (((strides[0] | strides[1] | strides[2]) * t.element_size() | t.data_ptr()) & 15)


def _rows(t: torch.Tensor) -> torch.Tensor:
    """(B,H,N,D) with a contiguous last dim and 16-byte aligned strides, copying only if needed."""
    return t if _aligned(t) else t.contiguous()


def _stream(t: torch.Tensor) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _problem(q, k, r_time, r_chan, sm_scale, window, q_time=(0, 0)) -> _nat.Problem:
    B, H, N, D = q.shape
    return _nat.Problem(B, H, k.shape[1], r_time.shape[-2], r_chan.shape[-2], D, int(window),
                        _dtype_code(q), float(sm_scale), 0, int(q_time[0]), int(q_time[1]))


def _launch_fwd(q, u, vt, z, k, r_time, r_chan, v, o, sm_scale, window, q_time, want_lse):
    """One `mvpa_fwd` call on tensors the kernels can read in place.  Returns the log-sum-exp (or None)."""
    lib = _nat.lib()
    prob = _problem(q, k, r_time, r_chan, sm_scale, window, q_time)
    lse = torch.empty((q.shape[0] * q.shape[1], q.shape[2]), device=q.device, dtype=torch.float32) if want_lse else None
    nbytes = lib.mvpa_fwd_workspace_bytes(ctypes.byref(prob))
    ws = torch.empty(nbytes, device=q.device, dtype=torch.uint8) if nbytes else None
    tq, tk, tv, to = _tensor(q), _tensor(k), _tensor(v), _tensor(o)
    with _nat.on_device(q.device):
        st = lib.mvpa_fwd(ctypes.byref(prob), ctypes.byref(tq), ctypes.byref(tk), ctypes.byref(tv),
                          u.data_ptr(), vt.data_ptr(), z.data_ptr(), r_time.data_ptr(), r_chan.data_ptr(),
                          ctypes.byref(to), None if lse is None else lse.data_ptr(), None if ws is None else ws.data_ptr(),
                          nbytes, _stream(q))
    _nat.check(st, "mvpa_fwd")
    if _CHECK_STATUS and nbytes:  # debugging aid: synchronises the stream
        _nat.check(lib.mvpa_workspace_status(ws.data_ptr(), nbytes, _stream(q)), "mvpa_fwd kernels")
    return lse


def _launch_bwd(q, u, vt, z, k, r_time, r_chan, v, o, lse, do, dq, dk, dv, sm_scale, window):
    """One `mvpa_bwd` call on tensors the kernels can read and write in place (dq, dk, dv are filled).  Returns the
    gradients of u, vt, z, r_time and r_chan, one after the other, flat, in q's dtype: they leave the library as fp32,
    and one buffer means that one cast serves all of them (every piece is a whole number of rows of D >= 16 elements,
    hence 16-byte aligned)."""
    lib = _nat.lib()
    prob = _problem(q, k, r_time, r_chan, sm_scale, window)
    sizes = [x.numel() for x in (u, vt, z, r_time, r_chan)]
    small = torch.empty(sum(sizes), device=q.device, dtype=torch.float32)
    ptrs, at = [], small.data_ptr()
    for n in sizes:
        ptrs.append(at)
        at += 4 * n
    nbytes = lib.mvpa_bwd_workspace_bytes(ctypes.byref(prob))
    ws = torch.empty(max(nbytes, 16), device=q.device, dtype=torch.uint8)
    T = [_tensor(x) for x in (q, k, v, o, do, dq, dk, dv)]
    r = [ctypes.byref(x) for x in T]
    with _nat.on_device(q.device):
        st = lib.mvpa_bwd(ctypes.byref(prob), r[0], r[1], r[2], u.data_ptr(), vt.data_ptr(),
                          z.data_ptr(), r_time.data_ptr(), r_chan.data_ptr(), r[3], lse.data_ptr(),
                          r[4], r[5], r[6], r[7], *ptrs, ws.data_ptr(), nbytes, _stream(q))
    _nat.check(st, "mvpa_bwd")
    if _CHECK_STATUS:  # debugging aid: synchronises the stream
        _nat.check(lib.mvpa_bwd_status(ctypes.byref(prob), ws.data_ptr(), nbytes, _stream(q)), "mvpa_bwd kernels")
    return small.to(q.dtype)


def _need_cuda(q):
    if not q.is_cuda:
        raise RuntimeError("flash_mvpa: tensors must be on a CUDA device (no CPU path)")


def _lay_out(q, u, vt, z, k, r_time, r_chan, v, q_time):
    """The operands as the kernels read them, copied only where their layout asks for it.  (They read through pointers: what
    does not go together is refused here.)"""
    _need_cuda(q)
    B, Hkv, N, D = shape = k.shape
    Bq, _, Nq, Dq = q.shape
    T, C = r_time.shape[-2], r_chan.shape[-2]
    row = Hkv * D
    if (v.shape != shape or Bq != B or Dq != D or T * C != N or Nq != (q_time[1] or T) * C or u.numel() != row or vt.numel() != row
            or z.numel() != row or r_time.numel() != row * T or r_chan.numel() != row * C):
        raise RuntimeError("flash_mvpa: the operands' shapes do not go together: "
                           + ", ".join(str(tuple(t.shape)) for t in (q, u, vt, z, k, r_time, r_chan, v)))
    dtype, device = q.dtype, q.get_device()
    if not (u.dtype is vt.dtype is z.dtype is k.dtype is r_time.dtype is r_chan.dtype is v.dtype is dtype
            and u.get_device() == vt.get_device() == z.get_device() == k.get_device() == r_time.get_device()
            == r_chan.get_device() == v.get_device() == device):
        raise RuntimeError("flash_mvpa: the operands are of different types or on different devices: "
                           + ", ".join(f"{t.dtype} {t.device}" for t in (q, u, vt, z, k, r_time, r_chan, v)))
    return (_rows(q), u.contiguous(), vt.contiguous(), z.contiguous(), _rows(k), r_time.contiguous(), r_chan.contiguous(),
            _rows(v))


class FlashMVPA(torch.autograd.Function):
    """Autograd wrapper; the counterpart of the reference's `FlashMVPA`
    (`attentions/attn.py:1013-1302`), taking the relative keys themselves instead of
    pre-multiplied score matrices.  The small tensors may have any shape with their elements in
    (kv head, row, D) order, r_time and r_chan with the rows next to last; their gradients take that shape."""

    @staticmethod
    def forward(ctx, q, u, vt, z, k, r_time, r_chan, v, sm_scale, window, q_time=(0, 0)):
        given = (q, u, vt, z, k, r_time, r_chan, v)
        ctx.sm_scale, ctx.window, ctx.q_time = sm_scale, window, q_time
        native = _host.module().forward(*given, sm_scale, window, *q_time, _CHECK_STATUS) if _host.usable(q) else None
        if native is not None:
            ctx.save_for_backward(*given, *native)
            ctx.copied = ()
            return native[0]
        q, u, vt, z, k, r_time, r_chan, v = read = _lay_out(*given, q_time)
        o = torch.empty_like(q)
        lse = _launch_fwd(q, u, vt, z, k, r_time, r_chan, v, o, sm_scale, window, q_time, True)
        ctx.save_for_backward(*read, o, lse)
        # what was copied, for second derivatives alone: the copy belongs to no graph
        ctx.copied = () if all(map(is_, given, read)) else [(i, t, t._version) for i, t in enumerate(given) if t is not read[i]]
        return o

    @staticmethod
    def backward(ctx, do):
        if ctx.q_time[1]:
            raise NotImplementedError("flash_mvpa: backward through a query time range is not implemented")
        if not torch.is_grad_enabled():
            return _gradients(do, *ctx.saved_tensors, ctx.sm_scale, ctx.window) + (None, None, None)
        # a graph of the gradient is wanted
        read = list(ctx.saved_tensors)
        for i, t, version in ctx.copied:
            if t.requires_grad:
                if t._version != version:
                    raise RuntimeError("flash_mvpa: an operand has been modified in place since the forward; its second "
                                       "derivative cannot be formed")
                read[i] = t.contiguous()
        return _FlashMVPAGrad.apply(do, *read, ctx.sm_scale, ctx.window) + (None, None, None)


def _gradients(do, q, u, vt, z, k, r_time, r_chan, v, o, lse, sm_scale, window):
    if _host.usable(q):
        native = _host.module().backward(do, q, u, vt, z, k, r_time, r_chan, v, o, lse, sm_scale, window, _CHECK_STATUS)
        if native is not None:
            return native
    # (a saved-tensor hook may have brought back any layout)
    q, u, vt, z, k, r_time, r_chan, v = _lay_out(q, u, vt, z, k, r_time, r_chan, v, (0, 0))
    o, lse = _rows(o), lse.contiguous()
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    small = _launch_bwd(q, u, vt, z, k, r_time, r_chan, v, o, lse, _rows(do), dq, dk, dv, sm_scale, window)
    shapes = [x.shape for x in (u, vt, z, r_time, r_chan)]
    sizes = [sh.numel() for sh in shapes]
    du, dvt, dz, drt, drc = (piece.view(sh) for piece, sh in zip(small.split(sizes), shapes))
    return dq, du, dvt, dz, dk, drt, drc, dv


class _FlashMVPAGrad(torch.autograd.Function):
    """The backward of `FlashMVPA` as a function of its own: the same kernels, and a derivative, taken in 64 bits on the
    materialised scores of one (sample, kv head) after the other.  Gradient penalties and Hessian products at sizes where
    (query heads per kv head, N, N) fits; the kernels have no second derivative."""

    @staticmethod
    def forward(ctx, do, *operands):
        ctx.save_for_backward(do, *operands[:8])
        ctx.sm_scale, ctx.window = operands[-2:]
        return tuple(t.clone() if t._is_view() else t for t in _gradients(do, *operands))

    @staticmethod
    def backward(ctx, *grads):
        create = torch.is_grad_enabled()
        with torch.enable_grad():
            ins = [t.view_as(t) if t.requires_grad else t for t in ctx.saved_tensors]
            q, k, T, C = ins[1], ins[5], ins[6].shape[-2], ins[7].shape[-2]
            (B, H, N, D), Hkv = q.shape, k.shape[1]
            rows = {0: N, 1: N, 5: N, 6: T, 7: C, 8: N}      # (the three biases: one row)

            def parts(t, i, b, j):   # what kv head j of sample b reads of operand i (or of its gradient), in 64 bits
                if i in (0, 1):
                    return t[b, j * (H // Hkv):(j + 1) * (H // Hkv)].double()
                return (t.reshape(B, Hkv, N, D)[b, j] if i in (5, 8) else t.reshape(Hkv, rows.get(i, 1), D)[j]).double()

            out = [[[None] * Hkv for _ in range(B)] for _ in ins]
            for b in range(B):
                for j in range(Hkv):
                    local = [parts(t, i, b, j) for i, t in enumerate(ins)]
                    local = [t if t.requires_grad else t.requires_grad_() for t in local]
                    o = _dense_head(*local[1:], ctx.sm_scale, ctx.window)
                    first = torch.autograd.grad(o, local[1:], local[0], create_graph=True)
                    inner = sum((f * parts(g, i + 1, b, j)).sum() for i, (f, g) in enumerate(zip(first, grads)))
                    for i, t in enumerate(torch.autograd.grad(inner, local, create_graph=create)):
                        out[i][b][j] = t
            res = []
            for i, t in enumerate(ins):
                if i in (0, 1):
                    whole = torch.stack([torch.cat(per_b) for per_b in out[i]])
                elif i in (5, 8):
                    whole = torch.stack([torch.stack(per_b) for per_b in out[i]])
                else:
                    whole = torch.stack([sum(per_b[j] for per_b in out[i]) for j in range(Hkv)])
                res.append(whole.reshape(t.shape).to(t.dtype))
        return (*res, None, None, None, None)


def _dense_head(q, u, vt, z, k, r_time, r_chan, v, sm_scale, window):
    """The operator for one kv head on materialised scores, in differentiable operations: q (heads, N, D), k, v (N, D)."""
    T, C = r_time.shape[0], r_chan.shape[0]
    n = torch.arange(T * C, device=q.device)
    t, c = n // C, n % C
    dt = t[:, None] - t[None, :]
    at = lambda x, index: x.gather(-1, index.expand(*x.shape[:-1], index.shape[-1]))
    s = (q + u) @ k.t()
    if window > 0:
        s = s.masked_fill((dt.abs() > window) & (t[:, None] != T - 1), 0.0)
    s = s + at((q + vt) @ r_time.t(), (T - 1 - dt).clamp(max=T - 1)) \
        + at((q + z) @ r_chan.t(), C - 1 - (c[:, None] - c[None, :]).abs())
    return torch.softmax((s * sm_scale).masked_fill(dt < 0, -math.inf), -1) @ v


def _attend(q, u, vt, z, k, r_time, r_chan, v, sm_scale, window, q_time):
    """FlashMVPA with or without its autograd record: a call that no gradient flows through goes to the kernels directly (and
    stores no log-sum-exp); whatever traces or transforms the call sees the autograd function.  (Most calls without a gradient
    never come here: see the start of `flash_mvpa`.)"""
    ts = (q, u, vt, z, k, r_time, r_chan, v)
    if ((torch.is_grad_enabled() and any(t.requires_grad for t in ts)) or not _nat.untraced()
            or not all(type(t) is torch.Tensor or type(t) is torch.nn.Parameter for t in ts)):
        return FlashMVPA.apply(*ts, sm_scale, window, q_time)
    q, u, vt, z, k, r_time, r_chan, v = _lay_out(*ts, q_time)
    o = torch.empty_like(q)
    _launch_fwd(q, u, vt, z, k, r_time, r_chan, v, o, sm_scale, window, q_time, False)
    return o


def flash_mvpa_into(out, q, u, vt, z, k, r_time, r_chan, v, sm_scale, window_size=10, q_time_range=None):
    """Inference form of `flash_mvpa`: no autograd record, no log-sum-exp output, and the result goes into
    `out`, a caller-owned (B,H,N,D) tensor that may be a strided view (e.g. a column block of the buffer the
    next projection reads).  u, vt, z (Hkv,D); r_time (Hkv,T,D); r_chan (Hkv,C,D).  `q_time_range=(t0, n)`:
    `q` and `out` hold only the tokens of time steps t0..t0+n-1 (see `flash_mvpa`).  No counterpart in the
    reference, whose operator always allocates its output (`attentions/attn.py:1047`)."""
    q_time = (0, 0) if q_time_range is None else (int(q_time_range[0]), int(q_time_range[1]))
    q, u, vt, z, k, r_time, r_chan, v = _lay_out(q, u, vt, z, k, r_time, r_chan, v, q_time)
    if not _aligned(out) or out.shape != q.shape or out.dtype != q.dtype or out.device != q.device:
        raise RuntimeError("flash_mvpa_into: `out` must have q's shape, type and device, a contiguous last dimension and 16-byte aligned strides")
    _launch_fwd(q, u, vt, z, k, r_time, r_chan, v, out, sm_scale, window_size, q_time, False)
    return out


def flash_mvpa(q, q_bias, q_btime, q_bchan, k_glob, k_time, k_chan, v, causal, sm_scale,
               window_size=0, p_drop=0.0, sequence_parallel=False, rel_bias_time=True,
               rel_bias_chan=True, generator=None, q_time_range=None):
    """Fused multi-variate parallel attention.

    q (B,H,N,D); q_bias/q_btime/q_bchan (1,Hkv,1,D) = u/v/z; k_glob, v (B,Hkv,N,D);
    k_time (1,Hkv,T,D); k_chan (1,Hkv,C,D); N == T*C, token n = t*C + c.  Returns o (B,H,N,D).

    As in the reference, causality is forced on whenever a relative term is used
    (`attentions/attn.py:1335-1336`) and the same shape checks raise
    (`:1339, 1344`).  `sequence_parallel` only chose a launch geometry in the
    reference (`:1165-1172`) and is accepted and ignored.  Structured attention dropout
    (`:1052-1062`) is applied to V on the way in (see below); runs with both relative terms off are
    not implemented and raise.

    `q_time_range=(t0, n)` (an extension, forward only): `q` holds only the tokens of time steps
    [t0, t0+n) while the keys, values and relative keys describe the whole sequence — what one
    rank computes when a long sample is sharded by query time blocks (`mvpa_shard`).
    """
    if rel_bias_time and rel_bias_chan and not p_drop and q_time_range is None and _host.usable(q):
        # an ordinary call that no gradient flows through, with nothing to refuse, copy or trace: one native call
        o = _host.module().attend(q, q_bias, q_btime, q_bchan, k_glob, k_time, k_chan, v, sm_scale, window_size, _CHECK_STATUS)
        if o is not None:
            return o
    if not (rel_bias_time or rel_bias_chan):
        raise NotImplementedError("flash_mvpa: at least one relative term is required (without them the "
                                  "reference runs a plain windowed attention, which these kernels are not)")
    # One term switched off: the reference kernels skip it and change nothing else
    # (`attentions/attn.py:187-216, 241-308`), which is the same attention with that term's relative key
    # at zero; its key and its query bias then receive zero gradients, as in the reference.
    if not rel_bias_time:
        k_time = k_time * 0
    if not rel_bias_chan:
        k_chan = k_chan * 0
    if p_drop and not 0 < p_drop < 1:
        raise ValueError(f"flash_mvpa: p_drop must be in [0, 1), got {p_drop}")
    q_heads, kv_heads = q.shape[1], v.shape[1]
    assert q_heads % kv_heads == 0, "Q heads must be divisible by KV heads."
    n_ctx, time_ctx, chan_ctx = k_glob.shape[2], k_time.shape[2], k_chan.shape[2]
    assert n_ctx == time_ctx * chan_ctx
    q_time = (0, 0)
    if q_time_range is not None:
        q_time = (int(q_time_range[0]), int(q_time_range[1]))
        assert q_time[1] > 0 and q.shape[2] == q_time[1] * chan_ctx
    else:
        assert q.shape[2] == n_ctx
    assert q.shape[-1] == k_glob.shape[-1] == v.shape[-1]
    assert q.shape[-1] in {16, 32, 64, 128}
    D = q.shape[-1]
    if p_drop and p_drop > 0:
        # Structured dropout of the reference (`attentions/attn.py:1052-1062, 316-321`): whole key time
        # steps and key channels are dropped, each with probability 1 - sqrt(1 - p_drop), and the kept
        # probabilities are divided by 1 - p_drop after the softmax denominator is taken.  The mask depends
        # on the key alone, so P_dropped V = (P (mask V)) / (1 - p_drop): one exact 0/1 pass over V before the
        # kernels and one fp32 scaling of their output (the reference divides P in fp32, `:235`), and autograd
        # carries both into dV and dO.  Same draws in the same order as the reference (channels, then time
        # steps), so a generator seeded alike gives the same mask.
        p_per_dim = 1 - math.sqrt(1 - p_drop)
        chan_keep = torch.rand(chan_ctx, device=q.device, generator=generator) > p_per_dim
        time_keep = torch.rand(time_ctx, device=q.device, generator=generator) > p_per_dim
        keep = (time_keep[:, None] & chan_keep[None, :]).reshape(1, 1, n_ctx, 1)
        v = v * keep.to(v.dtype)
    for x, n in ((q_bias, 1), (q_btime, 1), (q_bchan, 1), (k_time, time_ctx), (k_chan, chan_ctx)):
        if x.numel() != kv_heads * n * D:
            raise RuntimeError(f"flash_mvpa: shape {tuple(x.shape)} is invalid for {kv_heads} kv heads x {n} x {D}")
    if k_time.dim() != 4 or k_chan.dim() != 4:   # (the kernels' sizes are read off the axis next to the last)
        k_time, k_chan = k_time.reshape(1, kv_heads, time_ctx, D), k_chan.reshape(1, kv_heads, chan_ctx, D)
    o = _attend(q, q_bias, q_btime, q_bchan, k_glob, k_time, k_chan, v, sm_scale, window_size, q_time)
    if p_drop and p_drop > 0:
        o = (o.float() * (1.0 / (1 - p_drop))).to(o.dtype)
    return o
