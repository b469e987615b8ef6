"""GPU: the native calls of the parallel block where its surroundings or its modules are not the usual ones."""
import pytest
import torch

import models
from models import block_grad

pytestmark = pytest.mark.gpu


def _block(cuda, dtype=torch.float32, E=128, H=4, Hkv=2, I=160, B=2, T=13, C=5):
    torch.manual_seed(0)
    cfg = models.MVPFormerConfig(n_embd=E, n_layer=1, n_head=H, n_head_kv=Hkv, n_inner=I, attn_pdrop=0.0, resid_pdrop=0.0)
    block = models.MVPFormerBlock(cfg).to(cuda, dtype)
    r = lambda *s: torch.randn(*s, device=cuda).to(dtype).requires_grad_()
    return block, r(B, T, C, E), r(1, T, E), r(1, C, E)


def _inputs(block, x, pos, chan):
    return [x, pos, chan, *(p for n, p in block.named_parameters() if "ln_2" not in n)]


# a backward inside an autocast region that its forward was outside of
@pytest.mark.parametrize("dtype, region", [(torch.float32, torch.bfloat16), (torch.float32, torch.float16), (torch.bfloat16, torch.float16)])
def test_backward_inside_autocast(cuda, dtype, region):
    block, x, pos, chan = _block(cuda, dtype)
    ins = _inputs(block, x, pos, chan)
    y = block(x, pos, chan)[0]
    assert "BlockFunction" in type(y.grad_fn).__name__
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, ins, dy, retain_graph=True)
    graphed = torch.autograd.grad(y, ins, dy, retain_graph=True, create_graph=True)
    with torch.autocast("cuda", dtype=region):
        got = torch.autograd.grad(y, ins, dy, retain_graph=True)
        got_graphed = torch.autograd.grad(y, ins, dy, create_graph=True)
    for a, b, c, d in zip(want, got, graphed, got_graphed):
        assert a.dtype == b.dtype and torch.equal(a, b) and torch.equal(c, d)


def _resized(p, dim, by):
    shape = list(p.shape)
    shape[dim] += by
    return torch.nn.Parameter(torch.randn(shape, device=p.device).to(p.dtype))


# weights of other sizes than the block was made with, each alone: refused by the modules, and by the native call
@pytest.mark.parametrize("path, dim, by", [
    ("attn.q_attn.weight", 0, -32), ("attn.q_attn.weight", 0, 32), ("attn.c_attn.weight", 0, -32), ("attn.c_attn.weight", 0, 32),
    ("attn.position_net.weight", 0, -32), ("attn.channel_net.weight", 0, 32), ("attn.attn_bias", 0, -64), ("attn.attn_bias", 0, 32),
    ("attn.c_proj.weight", 1, -32), ("attn.c_proj.weight", 0, -32), ("mlp.gate_proj.weight", 0, 32), ("mlp.up_proj.weight", 0, -32),
    ("mlp.up_proj.weight", 0, 32), ("mlp.down_proj.weight", 1, -32), ("ln_1.weight", 0, -32)])
def test_resized_weights_are_refused(cuda, path, dim, by):
    block, x, pos, chan = _block(cuda)
    *way, last = path.split(".")
    owner = block.get_submodule(".".join(way))
    setattr(owner, last, _resized(getattr(owner, last), dim, by))
    with pytest.raises((RuntimeError, ValueError, AssertionError)):
        block(x, pos, chan)
    with pytest.raises(RuntimeError):
        block_grad.run(block, x, pos, chan)


# heads taken out of every projection that holds them, and of the counts: a smaller block, as before
def test_pruned_heads(cuda):
    block, x, pos, chan = _block(cuda)
    a = block.attn
    a.num_heads = 2
    a.q_attn.weight = torch.nn.Parameter(a.q_attn.weight[:64].clone())
    a.c_proj.weight = torch.nn.Parameter(a.c_proj.weight[:, :64].clone())
    y = block(x, pos, chan)[0]
    assert "BlockFunction" in type(y.grad_fn).__name__
    args = (x, pos, chan, block.ln_1.weight, a.q_attn.weight, a.c_attn.weight, a.position_net.weight, a.channel_net.weight, a.attn_bias,
            a.c_proj.weight, block.mlp.gate_proj.weight, block.mlp.up_proj.weight, block.mlp.down_proj.weight)
    want = block_grad.expression(*args, block.ln_1.eps, (2, 2, 32))
    assert (y - want).norm() <= 1e-5 * want.norm()


# what a saved-tensor hook brings back need not lie in memory as the kernels read it
@pytest.mark.parametrize("form", [lambda t: torch.nn.functional.pad(t, (0, 1))[..., :-1], lambda t: t.clone(),
                                  lambda t: torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape)])
def test_backward_of_rearranged_saved_tensors(cuda, form):
    block, x, pos, chan = _block(cuda)
    ins = _inputs(block, x, pos, chan)
    y = block(x, pos, chan)[0]
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, ins, dy)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), form):
        y = block(x, pos, chan)[0]
        assert "BlockFunction" in type(y.grad_fn).__name__
    for a, b in zip(torch.autograd.grad(y, ins, dy), want):
        assert (a - b).norm() <= 1e-5 * b.norm()


# the inference block inside autocast computes in the region's type throughout
def test_fused_branches_inside_autocast(cuda):
    block, x, _, _ = _block(cuda, B=2, T=13, C=5)
    x = x.detach().view(-1, 128)
    rt, rc = torch.randn(2, 13, 32, device=cuda), torch.randn(2, 5, 32, device=cuda)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got = [block.fused_branches(x, a, b, 2, 13, 5) for a, b in ((rt, rc), (rt.bfloat16(), rc.bfloat16()))]
        again = block.fused_branches(x.bfloat16(), rt.bfloat16(), rc.bfloat16(), 2, 13, 5)
    want = block.bfloat16().fused_branches(x.bfloat16(), rt.bfloat16(), rc.bfloat16(), 2, 13, 5)
    for y in (*got, again):
        assert y.dtype == torch.bfloat16 and torch.equal(y, want)


def test_without_the_extension(cuda, monkeypatch):
    import attentions
    import mvpa_host
    block, x, pos, chan = _block(cuda)
    ins = _inputs(block, x, pos, chan)
    gen = torch.Generator().manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=gen).to(cuda)
    a = [r(2, 4, 30, 64), r(1, 2, 1, 64), r(1, 2, 1, 64), r(1, 2, 1, 64), r(2, 2, 30, 64), r(1, 2, 5, 64), r(1, 2, 6, 64), r(2, 2, 30, 64)]
    y = block(x, pos, chan)[0]
    dy = torch.randn_like(y)
    want, o = torch.autograd.grad(y, ins, dy), attentions.flashmvpa(*a, True, 0.125, window_size=10)

    def refuse(force=False):
        raise ImportError("no compiler")

    monkeypatch.setattr(mvpa_host, "_module", None)
    monkeypatch.setattr(mvpa_host, "_refused", False)
    monkeypatch.setattr(mvpa_host, "build", refuse)
    with pytest.warns(RuntimeWarning, match="no compiler"):
        assert torch.equal(attentions.flashmvpa(*a, True, 0.125, window_size=10), o)
    y2 = block(x, pos, chan)[0]
    assert "BlockFunction" not in type(y2.grad_fn).__name__ and (y2 - y).norm() <= 1e-5 * y.norm()
    for g, w in zip(torch.autograd.grad(y2, ins, dy), want):
        assert (g - w).norm() <= 1e-5 * w.norm()
