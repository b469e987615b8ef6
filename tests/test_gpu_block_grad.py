"""GPU: gradients of gradients through the operator and the one-function block, against 64-bit dense torch and against the
modules, and the blocks that must keep going through their modules."""
import pytest
import torch
import torch.nn.functional as F

import attentions
import layers.mvpa as layer_module
import models
import mvpa_port_torch as port
from models import mvpformer

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm()).item()


def _one_function(out):
    return "BlockFunction" in type(out.grad_fn).__name__


class _Stack(torch.nn.Module):
    """Blocks that share non-leaf time and channel embeddings, as the model's do."""

    def __init__(self, n, E=64, H=4, Hkv=2, I=80, **rates):
        super().__init__()
        cfg = models.MVPFormerConfig(n_embd=E, n_layer=n, n_head=H, n_head_kv=Hkv, n_inner=I, n_positions=16, n_channels=16,
                                     attn_pdrop=0.0, resid_pdrop=0.0)
        self.h = torch.nn.ModuleList([models.MVPFormerBlock(cfg) for _ in range(n)])
        self.pos, self.chan = torch.nn.Embedding(16, E), torch.nn.Embedding(16, E)
        for name, p in self.named_parameters():
            torch.nn.init.normal_(p, mean=1.0 if "ln_" in name else 0.0, std=0.15)

    def embeddings(self, T, C):
        dev = self.pos.weight.device
        return self.pos(torch.arange(T, device=dev))[None], self.chan(torch.arange(C, device=dev))[None]

    def forward(self, x):
        pos, chan = self.embeddings(x.shape[1], x.shape[2])
        for block in self.h:
            x = block(x, pos, chan)[0]
        return x

    def used(self):
        return [p for n, p in self.named_parameters() if "ln_2" not in n]


def _stack64(stack, x):
    """The same in plain torch at the inputs' precision, dense attention; nothing of the package's arithmetic."""
    pos, chan = stack.embeddings(x.shape[1], x.shape[2])
    B, T, C, E = x.shape
    N = T * C
    for block in stack.h:
        a, m = block.attn, block.mlp
        H, Hkv, D = a.num_heads, a.num_kv_heads, a.head_dim
        xn = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + block.ln_1.eps) * block.ln_1.weight
        q = F.linear(xn, a.q_attn.weight).view(B, N, H, D).transpose(1, 2)
        k, v = (t.transpose(1, 2) for t in F.linear(xn, a.c_attn.weight).view(B, N, 2 * Hkv, D).split(Hkv, dim=2))
        rt = F.linear(pos, a.position_net.weight).view(T, Hkv, D).transpose(0, 1)
        rc = F.linear(chan, a.channel_net.weight).view(C, Hkv, D).transpose(0, 1)
        u, vt, z = (b.view(Hkv, D) for b in a.attn_bias.split(Hkv * D))
        o = port.rel_attn(q, u, vt, z, k, rt, rc, v, D ** -0.5, 10).transpose(1, 2).reshape(B, T, C, E)
        mlp = F.linear(F.silu(F.linear(xn, m.gate_proj.weight)) * F.linear(xn, m.up_proj.weight), m.down_proj.weight)
        x = x + mlp + F.linear(o, a.c_proj.weight)
    return x


def _hook(stack):
    return [b.mlp.register_forward_hook(lambda *a: None) for b in stack.h]


# fp32 products in another order, three blocks deep
def test_graph_of_the_gradient_stops_at_each_block(cuda):
    torch.manual_seed(0)
    stack = _Stack(3).to(cuda)
    x = torch.randn(2, 13, 5, 64, device=cuda, requires_grad=True)
    dy = torch.randn(2, 13, 5, 64, device=cuda)
    ins = [x, *stack.used()]
    y = stack(x)
    assert _one_function(y)
    plain = torch.autograd.grad(y, ins, dy, retain_graph=True)
    graphed = torch.autograd.grad(y, ins, dy, create_graph=True)
    handles = _hook(stack)
    y2 = stack(x)
    assert not _one_function(y2)
    ref = torch.autograd.grad(y2, ins, dy)
    for h in handles:
        h.remove()
    for a, b, c in zip(plain, graphed, ref):
        assert _rel(a, c) <= 1e-5 and _rel(b, c) <= 1e-5


# The derivative of a gradient penalty with respect to everything, through two blocks, on both routes.  fp32 against 64 bits:
# a chain of a few dozen products, each of at most 80 terms rounded to 2^-24 and each condition number of order one.
@pytest.mark.parametrize("hooked", [False, True])
def test_gradient_penalty_against_64_bits(cuda, hooked):
    torch.manual_seed(1)
    stack = _Stack(2).to(cuda)
    x = torch.randn(1, 13, 3, 64, device=cuda, requires_grad=True)
    dy = torch.randn(1, 13, 3, 64, device=cuda)

    def penalty_gradients(f, mod, x, dy):
        ins = [x, *mod.used()]
        first = torch.autograd.grad(f(x), ins, dy, create_graph=True)
        return torch.autograd.grad(sum((g * g).sum() for g in first), ins)

    handles = _hook(stack) if hooked else []
    got = penalty_gradients(stack, stack, x, dy)
    for h in handles:
        h.remove()
    s64 = _Stack(2).to(cuda).double()
    s64.load_state_dict({k: v.double() for k, v in stack.state_dict().items()})
    want = penalty_gradients(lambda t: _stack64(s64, t), s64, x.detach().double().requires_grad_(), dy.double())
    for a, b in zip(got, want):
        assert _rel(a, b) <= 2e-5


def _operands(B, H, Hkv, T, C, D, dtype, cuda, strided):
    g = torch.Generator().manual_seed(T * 100 + C)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).to(dtype).to(cuda)
    N = T * C
    a = [r(B, H, N, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(B, Hkv, N, D), r(1, Hkv, T, D), r(1, Hkv, C, D),
         r(B, Hkv, N, D)]
    if strided:   # token-major storage (read in place), and an odd row stride and reversed axes (copied)
        a[0] = a[0].transpose(1, 2).contiguous().transpose(1, 2)
        a[4] = torch.cat([a[4], a[4][..., :1]], -1)[..., :D]
        a[5] = a[5].transpose(1, 2).contiguous().transpose(1, 2)
    return a, r(B, H, N, D)


# One head, several, grouped; one time step, steps beyond the window (masked content), one channel.  16-bit types: the
# first derivatives are rounded once (2^-8, 2^-11) before they are squared, and the result once more.
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])
@pytest.mark.parametrize("shape,strided", [((1, 1, 1, 1, 3, 16), False), ((2, 4, 2, 14, 3, 32), True), ((1, 2, 1, 15, 1, 64), False)])
def test_operator_second_derivative(cuda, dtype, tol, shape, strided):
    args, do = _operands(*shape, dtype, cuda, strided)
    D = shape[-1]

    def second(f, args, do):
        ins = [t.detach().requires_grad_() for t in (*args, do)]
        first = torch.autograd.grad(f(*ins[:-1]), ins[:-1], ins[-1], create_graph=True)
        return torch.autograd.grad(sum((g.double() * g).sum() for g in first), ins)

    got = second(lambda *a: attentions.flashmvpa(*a, True, D ** -0.5, window_size=10), args, do)
    want = second(lambda *a: port.rel_attn(*a, D ** -0.5, 10), [t.double() for t in args], do.double())
    for a, t, b in zip(got, (*args, do), want):
        assert a.dtype == dtype and a.shape == t.shape
        assert (a.double() - b).norm() <= tol * max(b.norm().item(), 1.0)


def _block(cuda, E=64, H=4, Hkv=2):
    torch.manual_seed(0)
    stack = _Stack(1, E=E, H=H, Hkv=Hkv).to(cuda)
    pos, chan = stack.embeddings(6, 5)
    return stack.h[0], torch.randn(1, 6, 5, E, device=cuda), pos, chan


def test_replaced_code_is_not_bypassed(cuda, monkeypatch):
    block, x, pos, chan = _block(cuda)
    assert _one_function(block(x, pos, chan)[0])
    calls = []

    def seen(f):
        def g(*a, **k):
            calls.append(f)
            return f(*a, **k)
        return g

    for owner, name in ((mvpformer.RMSNorm, "forward"), (mvpformer.LlamaMLP, "forward"), (torch.nn.Linear, "forward"),
                        (torch.nn.Dropout, "forward"), (layer_module.MVPFormerGQAFlashAttention, "forward"),
                        (layer_module.MVPFormerGQAAttention, "_mvpa_forward"), (layer_module, "flashmvpa")):
        with monkeypatch.context() as m:
            m.setattr(owner, name, seen(getattr(owner, name)))
            calls.clear()
            assert not _one_function(block(x, pos, chan)[0]) and calls, (owner, name)
    with monkeypatch.context() as m:
        m.setattr(block.attn, "_mvpa_forward", seen(block.attn._mvpa_forward))
        calls.clear()
        assert not _one_function(block(x, pos, chan)[0]) and calls
    assert _one_function(block(x, pos, chan)[0])


def test_recording_modes_see_the_operations(cuda):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Ops(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Calls(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))

    block, x, pos, chan = _block(cuda)
    for mode in (Ops, Calls):
        seen = []
        with mode():
            y = block(x, pos, chan)[0]
        assert not _one_function(y)
        assert any("silu" in s for s in seen) and any("rsqrt" in s for s in seen) and any("pow" in s for s in seen)
    with torch.device(cuda):   # a default device is a function mode too, but watches nothing
        assert _one_function(block(x, pos, chan)[0])


@pytest.mark.parametrize("E,H,Hkv", [(96, 2, 1), (96, 6, 4)])   # head_dim 48; query heads that no kv head divides
def test_refused_heads_are_refused_alike(cuda, E, H, Hkv):
    block, x, pos, chan = _block(cuda, E=E, H=H, Hkv=Hkv)
    with pytest.raises(AssertionError):
        block(x, pos, chan)


def test_outputs_and_gradients_may_be_changed_in_place(cuda):
    import mvpa_ops
    block, x, pos, chan = _block(cuda)
    w = block.ln_1.weight
    for f in (lambda t: block(t, pos, chan)[0], block.ln_1, lambda t: mvpa_ops.swiglu(t, t + 1)):
        y, z = f(x.requires_grad_()), f(x)
        y.mul_(2).add_(x.detach())
        y.view(-1)[3] = 0
        z = (z * 2 + x.detach()) * (torch.arange(z.numel(), device=cuda) != 3).view(z.shape)
        assert torch.equal(y, z)
        for a, b in zip(torch.autograd.grad(y.sum(), (x, w), allow_unused=True), torch.autograd.grad(z.sum(), (x, w), allow_unused=True)):
            assert (a is None and b is None) or torch.equal(a, b)
    args, do = _operands(1, 2, 1, 5, 3, 16, torch.float32, cuda, False)
    ins = [t.requires_grad_() for t in args]
    o = attentions.flashmvpa(*ins, True, 0.25, window_size=10)
    for t, g in zip(ins, torch.autograd.grad(o, ins, do, create_graph=True)):
        assert g.mul_(2).shape == t.shape
    for g in torch.autograd.grad(block(x, pos, chan)[0].sum(), (x, w)):
        g.mul_(w.sum())
