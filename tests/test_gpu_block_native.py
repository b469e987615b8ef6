"""GPU: the native calls of the parallel block where its surroundings or its modules are not the usual ones."""
import pytest
import torch

import models

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
