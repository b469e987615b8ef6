"""GPU: the one-function block against the modules where a graph of the gradient is built."""
import pytest
import torch

import models

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
