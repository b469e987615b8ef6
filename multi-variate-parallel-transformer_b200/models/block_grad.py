"""Training form of the parallel block (`models/mvpformer.py:132-147`, h = x + MLP(ln_1 x) + Attn(ln_1 x)) as ONE autograd
function.

The same operations as the modules run, in the same order, but with what lies between them removed: the residual and
branch sums are accumulated by the output projections (beta = 1 products instead of two additions), the four
projections' input gradients by their products (instead of three additions), the residual's gradient by the RMSNorm
backward kernel; the attention backward writes dq, dk, dv straight into the buffers the weight-gradient products read
(no slices, concatenations or copies), and autograd keeps one node per block instead of about forty.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

import layers.mvpa as _layer
import mvpa_host as _host
import mvpa_native as _nat
import mvpa_ops
from attentions import attn as _attn
from attentions import flashmvpa

WINDOW = 10


def expression(x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd, eps, heads):
    """The block in differentiable operations (what a graph of the gradient is built from)."""
    H, Hkv, D = heads
    B, T, C, E = x.shape
    N, KV = T * C, Hkv * D
    xn = mvpa_ops.rmsnorm_train(x, ln_w, eps)
    q = F.linear(xn, wq).view(B, N, H, D).permute(0, 2, 1, 3)
    k, v = (t.permute(0, 2, 1, 3) for t in F.linear(xn, wkv).view(B, N, 2 * Hkv, D).split(Hkv, dim=2))
    rt = F.linear(pos, wpos).view(1, T, Hkv, D).permute(0, 2, 1, 3)
    rc = F.linear(chan, wchan).view(1, C, Hkv, D).permute(0, 2, 1, 3)
    u, vt, z = (b.view(1, Hkv, 1, D) for b in bias.clone().split(KV))    # (what a saved-tensor hook brought back may lie anywhere)
    o = flashmvpa(q, u, vt, z, k, rt, rc, v, causal=True, sm_scale=1.0 / (D ** 0.5), window_size=WINDOW)
    mlp = F.linear(mvpa_ops.swiglu(F.linear(xn, wg), F.linear(xn, wu)), wd)
    return x + mlp + F.linear(o.permute(0, 2, 1, 3).reshape(B, T, C, H * D), wc)


def through_expression(f, ins, need, grad_out):
    """Gradients of f(*ins) for `grad_out`, differentiable if gradients are recorded; None where `need` is False.
    They are taken with respect to aliases of `ins`: an input's own history may lead to another input (a later block's x
    depends on the embeddings that it also receives), and autograd would follow it and return total derivatives."""
    create = torch.is_grad_enabled()
    with torch.enable_grad():
        local = [t.view_as(t) if t.requires_grad else t.detach().requires_grad_(n) for t, n in zip(ins, need)]
        got = iter(torch.autograd.grad(f(*local), [t for t, n in zip(local, need) if n], grad_out, create_graph=create))
    return [next(got) if n else None for n in need]


class BlockFunction(torch.autograd.Function):
    """Forward and backward are one native call each (`csrc_host/mvpa_host.cpp`: block_forward, block_backward)."""

    @staticmethod
    def forward(ctx, x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd, eps, heads):
        given = (x, pos, chan, ln_w, wq, wkv, wpos, wchan, bias, wc, wg, wu, wd)
        got = _host.module().block_forward(*given, eps, WINDOW, *heads, _attn._CHECK_STATUS)
        if got is None:
            raise RuntimeError("block: tensors that the kernels cannot take in place")   # (`applies` has looked at them)
        ctx.save_for_backward(*given, *got[1:])      # ... xn, q, kv, g, up, rt, rc, o, lse, act
        ctx.eps, ctx.heads = eps, heads
        return got[0]

    @staticmethod
    def backward(ctx, dh):
        saved = ctx.saved_tensors
        need = ctx.needs_input_grad[:13]
        if not torch.is_grad_enabled() and _nat.untraced() and mvpa_ops._plain(dh.contiguous()):
            mask = sum(n << i for i, n in enumerate(need))
            grads = _host.module().block_backward(dh, *saved, mask, ctx.eps, WINDOW, *ctx.heads, _attn._CHECK_STATUS)
            if grads is not None:
                return (*grads, None, None)
        # a graph of the gradient is wanted (or a transform is active): through the differentiable operations, in the forward's types
        with torch.autocast("cuda", enabled=False):
            grads = through_expression(lambda *ins: expression(*ins, ctx.eps, ctx.heads), saved[:13], need, dh)
        return (*grads, None, None)


def shipped(cls):
    """A module class with the code that it came with; a later replacement of its `forward` shows against it."""
    return cls, cls.forward


_LINEAR, _DROPOUT = shipped(torch.nn.Linear), shipped(torch.nn.Dropout)
_ATTENTION = _layer.MVPFormerGQAAttention._mvpa_forward


def _unhooked(m, code):
    cls, forward = code
    return (type(m) is cls and cls.forward is forward and "forward" not in m.__dict__ and not m._forward_hooks
            and not m._forward_pre_hooks and not m._backward_hooks and not m._backward_pre_hooks)


def applies(block, x, pos, chan, classes) -> bool:
    """Whether `block` is exactly the computation above on tensors the kernels take in place: the shipped modules (norm,
    attention and MLP in `classes`, as `shipped` returned them), neither they nor their code replaced, hooked or patched,
    no dropout or autocast, weights of the sizes that go together, one dtype, contiguous and 16-byte aligned, and nothing
    tracing the call.  Everything else goes
    through the modules."""
    norm, attn, mlp = classes
    a, m = block.attn, block.mlp
    if not (_unhooked(block.ln_1, norm) and _unhooked(a, attn) and _unhooked(m, mlp)):
        return False
    if getattr(a._mvpa_forward, "__func__", None) is not _ATTENTION or _layer.flashmvpa is not flashmvpa:
        return False
    linears = (a.q_attn, a.c_attn, a.position_net, a.channel_net, a.c_proj, m.gate_proj, m.up_proj, m.down_proj)
    if not all(_unhooked(l, _LINEAR) and l.bias is None for l in linears):
        return False
    for d in (a.attn_dropout, a.resid_dropout):
        if not _unhooked(d, _DROPOUT) or (d.training and d.p):
            return False
    if a.training and a.attn_dropout.p or torch.nn.modules.module._has_any_global_hook() or torch.is_autocast_enabled("cuda"):
        return False
    if a.head_dim not in (16, 32, 64, 128) or a.num_heads % a.num_kv_heads:
        return False                 # (what the operator refuses is refused by the operator)
    if not _host.usable(x):
        return False                 # (without the extension there is no function, but the modules)
    if x.dim() != 4 or pos.shape != (1, x.shape[1], x.shape[3]) or chan.shape != (1, x.shape[2], x.shape[3]):
        return False
    # (weights of other sizes than the module was made with: a pruned head, a replaced projection)
    weights = [l.weight for l in linears]
    E, Q, KV, I = x.shape[3], a.num_heads * a.head_dim, a.num_kv_heads * a.head_dim, weights[5].shape[0]
    if ([w.shape for w in weights] != [(Q, E), (2 * KV, E), (KV, E), (KV, E), (E, Q), (I, E), (I, E), (E, I)]
            or block.ln_1.weight.shape != (E,) or a.attn_bias.numel() != 3 * KV):
        return False
    ts = (x, pos, chan, block.ln_1.weight, a.attn_bias, *weights)
    return (mvpa_ops._plain(*ts) and mvpa_ops._rows_fit(x) and I * x.element_size() % 16 == 0
            and any(t.requires_grad for t in ts))


def run(block, x, pos, chan):
    a, m = block.attn, block.mlp
    return BlockFunction.apply(x, pos, chan, block.ln_1.weight, a.q_attn.weight, a.c_attn.weight, a.position_net.weight,
                               a.channel_net.weight, a.attn_bias, a.c_proj.weight, m.gate_proj.weight, m.up_proj.weight,
                               m.down_proj.weight, block.ln_1.eps, (a.num_heads, a.num_kv_heads, a.head_dim))
