"""GPU: the differentiable RMSNorm and SwiGLU of the training path at the edges of their launch shapes, against torch in
64 bits, and the routes that torch expressions keep serving."""
import pytest
import torch

import mvpa_ops

pytestmark = pytest.mark.gpu

# fp32: sums of up to 4096 terms in the norm, three units in the last place (2^-23) without sums in SwiGLU; bf16 (unit roundoff
# 2^-8): one rounding of the result around fp32 arithmetic, and for SwiGLU a second one, of silu(gate) before the product,
# as eager PyTorch does
TOL = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -8}
TOL_SWIGLU = {torch.float32: 3 * 2.0 ** -23, torch.bfloat16: 2 * 2.0 ** -8}


def _rel(got, want):
    return (got.double() - want).norm() / want.norm()


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


@pytest.mark.parametrize("dtype,rows,width", [(torch.bfloat16, 1, 8), (torch.bfloat16, 9, 768), (torch.bfloat16, 5000, 768),
                                              (torch.bfloat16, 33, 4096), (torch.float32, 7, 4), (torch.float32, 2500, 260),
                                              (torch.float32, 40, 2048)])
def test_rmsnorm_gradients(cuda, dtype, rows, width):
    g = torch.Generator().manual_seed(rows + width)
    x, dy = (torch.randn(rows, width, generator=g).to(dtype).to(cuda) for _ in range(2))
    w = (1 + 0.1 * torch.randn(width, generator=g)).to(dtype).to(cuda)
    a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
    y = mvpa_ops.rmsnorm_train(a, b, 1e-5)
    assert "RMSNorm" in type(y.grad_fn).__name__
    got = (y,) + torch.autograd.grad(y, (a, b), dy)
    a64, b64 = x.double().requires_grad_(), w.double().requires_grad_()
    y64 = _norm64(a64, b64, 1e-5)
    for v, ref in zip(got, (y64,) + torch.autograd.grad(y64, (a64, b64), dy.double())):
        assert v.dtype == dtype and _rel(v, ref) <= TOL[dtype]


@pytest.mark.parametrize("dtype,shape", [(torch.bfloat16, (1, 8)), (torch.bfloat16, (3, 7, 1728)), (torch.float32, (5, 4)),
                                         (torch.float32, (2, 300, 516))])
def test_swiglu_gradients(cuda, dtype, shape):
    g = torch.Generator().manual_seed(len(shape))
    gate, up, dy = (torch.randn(*shape, generator=g).to(dtype).to(cuda) for _ in range(3))
    a, b = gate.clone().requires_grad_(), up.clone().requires_grad_()
    y = mvpa_ops.swiglu(a, b)
    assert "SwiGLU" in type(y.grad_fn).__name__
    got = (y,) + torch.autograd.grad(y, (a, b), dy)
    a64, b64 = gate.double().requires_grad_(), up.double().requires_grad_()
    y64 = torch.nn.functional.silu(a64) * b64
    for v, ref in zip(got, (y64,) + torch.autograd.grad(y64, (a64, b64), dy.double())):
        assert v.dtype == dtype and _rel(v, ref) <= TOL_SWIGLU[dtype]


# fp32, element by element, gates as large as a trained MLP's: an exponential and a division within one unit in the last
# place each (2^-23 relative), the addition and the products half a unit each: three units for silu(gate) * up.  dgate's
# factor 1 + gate (1 - s) cancels near gate = -1.28, so it is held in the 2-norm: exp's unit times gate, of size std.
@pytest.mark.parametrize("std", [1.0, 3.0, 8.0])
def test_fp32_elementwise_accuracy(cuda, std):
    g = torch.Generator().manual_seed(3)
    gate, up, dy = (torch.randn(300, 1028, generator=g).to(cuda) for _ in range(3))
    gate = (gate * std).requires_grad_()
    up.requires_grad_()
    y = mvpa_ops.swiglu(gate, up)
    dgate, dup = torch.autograd.grad(y, (gate, up), dy)
    a64, b64 = gate.detach().double().requires_grad_(), up.detach().double().requires_grad_()
    y64 = torch.nn.functional.silu(a64) * b64
    dgate64, dup64 = torch.autograd.grad(y64, (a64, b64), dy.double())
    ulp = 2.0 ** -23
    worst = lambda v, r: ((v.double() - r).abs() / r.abs().clamp_min(2.0 ** -100)).max().item()
    assert worst(y, y64) <= 3 * ulp and worst(dup, dup64) <= 3 * ulp
    assert _rel(dgate, dgate64) <= max(1.0, std / 3) * ulp


# The norm's weight gradient sums over the rows; its terms are products of values with about half a unit of error each, and
# their sum may add no more than that again.
@pytest.mark.parametrize("rows,width", [(2000, 260), (300, 768), (40, 2048)])
def test_fp32_norm_accuracy(cuda, rows, width):
    g = torch.Generator().manual_seed(5)
    x, dy = (torch.randn(rows, width, generator=g).to(cuda) for _ in range(2))
    w = (1 + 0.1 * torch.randn(width, generator=g)).to(cuda)
    ins = [x.requires_grad_(), w.requires_grad_()]
    y = mvpa_ops.rmsnorm_train(*ins, 1e-5)
    got = (y, *torch.autograd.grad(y, ins, dy))
    ins64 = [t.detach().double().requires_grad_() for t in ins]
    y64 = _norm64(*ins64, 1e-5)
    for v, r in zip(got, (y64, *torch.autograd.grad(y64, ins64, dy.double()))):
        assert _rel(v, r) <= 2.0 ** -23


def test_second_derivatives_and_transforms(cuda):
    x = torch.randn(6, 64, device=cuda, requires_grad=True)
    w = torch.randn(64, device=cuda, requires_grad=True)

    def second(f, *args):
        g = torch.autograd.grad(f(*args).pow(2).sum(), args, create_graph=True)
        return torch.autograd.grad(sum(t.pow(2).sum() for t in g), args)

    ref = lambda a, b: _norm64(a, b, 1e-5)
    for v, r in zip(second(lambda a, b: mvpa_ops.rmsnorm_train(a, b, 1e-5), x, w), second(ref, x, w)):
        torch.testing.assert_close(v, r, rtol=1e-4, atol=1e-4)
    u = torch.randn(6, 64, device=cuda, requires_grad=True)
    for v, r in zip(second(mvpa_ops.swiglu, x, u), second(lambda a, b: torch.nn.functional.silu(a) * b, x, u)):
        torch.testing.assert_close(v, r, rtol=1e-4, atol=1e-4)
    one = torch.ones(64, device=cuda)
    _, t1 = torch.func.jvp(lambda a: mvpa_ops.rmsnorm_train(a, one, 1e-5), (x.detach(),), (x.detach(),))
    _, t2 = torch.func.jvp(lambda a: _norm64(a, one, 1e-5), (x.detach(),), (x.detach(),))
    torch.testing.assert_close(t1, t2)
    # a batch of incoming gradients, and inputs the kernels do not take (layout, width, type)
    y = mvpa_ops.rmsnorm_train(x, w, 1e-5)
    eye = torch.randn(3, 6, 64, device=cuda)
    batched = torch.autograd.grad(y, x, eye, is_grads_batched=True, retain_graph=True)[0]
    torch.testing.assert_close(batched[1], torch.autograd.grad(y, x, eye[1])[0], rtol=1e-5, atol=1e-5)
    xt = torch.randn(64, 6, device=cuda).t()
    torch.testing.assert_close(mvpa_ops.rmsnorm_train(xt, w, 1e-5), _norm64(xt, w, 1e-5))
    odd = torch.randn(4, 7, device=cuda)
    torch.testing.assert_close(mvpa_ops.rmsnorm_train(odd, odd[0], 1e-5), _norm64(odd, odd[0], 1e-5))
    h = torch.randn(4, 16, device=cuda, dtype=torch.float16)
    torch.testing.assert_close(mvpa_ops.swiglu(h, h), torch.nn.functional.silu(h) * h)


def _block(cuda, dtype, E=128, H=4, Hkv=2, I=176, T=13, C=10, B=2):
    import models
    torch.manual_seed(0)
    cfg = models.MVPFormerConfig(n_embd=E, n_layer=1, n_head=H, n_head_kv=Hkv, n_inner=I, n_positions=16, n_channels=16,
                                 attn_pdrop=0.0, resid_pdrop=0.0)
    block = models.MVPFormerBlock(cfg).to(cuda).to(dtype)
    for p in block.parameters():
        torch.nn.init.normal_(p, std=0.1)
    x, pos, chan = (torch.randn(*s, E, device=cuda).to(dtype).requires_grad_() for s in ((B, T, C), (1, T), (1, C)))
    return block, x, pos, chan, torch.randn(B, T, C, E, device=cuda).to(dtype)


# The one-function block against the modules, which an (empty) hook brings back.  fp32: the same products in another
# order; bf16: one rounding per intermediate result (2^-9 each, about six on the longest way) on both sides.
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 3e-2)])
@pytest.mark.parametrize("frozen", [False, True])
def test_block_function_equals_the_modules(cuda, dtype, tol, frozen):
    block, x, pos, chan, dy = _block(cuda, dtype)
    if frozen:
        for m in (block.attn.q_attn, block.mlp.down_proj, block.ln_1):
            m.weight.requires_grad_(False)
        pos.requires_grad_(False)
    ins = [t for n, t in [("x", x), ("pos", pos), ("chan", chan), *block.named_parameters()]
           if t.requires_grad and not n.startswith("ln_2")]
    y = block(x, pos, chan)[0]
    assert "BlockFunction" in type(y.grad_fn).__name__
    got = (y,) + torch.autograd.grad(y, ins, dy)
    handle = block.mlp.register_forward_hook(lambda *a: None)
    y2 = block(x, pos, chan)[0]
    assert "BlockFunction" not in type(y2.grad_fn).__name__
    ref = (y2,) + torch.autograd.grad(y2, ins, dy)
    handle.remove()
    for a, b in zip(got, ref):
        assert a.dtype == b.dtype and a.shape == b.shape and _rel(a, b.double()) <= tol


def test_block_function_graph_of_the_gradient_and_other_routes(cuda):
    block, x, pos, chan, dy = _block(cuda, torch.float32)

    def penalty(out):
        return torch.autograd.grad(out, x, dy, create_graph=True)[0].pow(2).sum()

    p1 = penalty(block(x, pos, chan)[0])
    g1 = torch.autograd.grad(p1, block.mlp.up_proj.weight)[0]
    handle = block.mlp.register_forward_hook(lambda *a: None)
    p2 = penalty(block(x, pos, chan)[0])
    g2 = torch.autograd.grad(p2, block.mlp.up_proj.weight)[0]
    handle.remove()
    assert _rel(p1, p2.double()) <= 1e-5 and _rel(g1, g2.double()) <= 1e-4
    block.attn.resid_dropout.p = 0.5
    assert "BlockFunction" not in type(block(x, pos, chan)[0].grad_fn).__name__
    block.eval()
    assert "BlockFunction" in type(block(x, pos, chan)[0].grad_fn).__name__
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert "BlockFunction" not in type(block(x, pos, chan)[0].grad_fn).__name__
