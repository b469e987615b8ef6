"""GPU: the native host path of the operator and the block against the Python path around the same kernels: the same bits
for every form it accepts, and what it does not take (or what is refused) goes as before."""
import pytest
import torch

import attentions
import models
import mvpa_host
from models.mvpformer import MVPFormerBlock

pytestmark = pytest.mark.gpu


def _operands(cuda, dtype, B=2, H=4, Hkv=2, T=5, C=6, D=64, seed=0):
    gen = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=gen).to(cuda, dtype)
    return [r(B, H, T * C, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(B, Hkv, T * C, D), r(1, Hkv, T, D),
            r(1, Hkv, C, D), r(B, Hkv, T * C, D)]


def _permuted(t):    # (B, heads, N, D) as a view of (B, N, heads, D)
    return t.transpose(1, 2).contiguous().transpose(1, 2)


def _padded(t):      # rows of a wider buffer: strides that are no products of the sizes, still 16-byte aligned
    return torch.nn.functional.pad(t, (0, 16))[..., :t.shape[-1]]


def _odd(t):         # strides that the kernels cannot take: copied on the way in
    return torch.nn.functional.pad(t, (0, 1))[..., :t.shape[-1]]


FORMS = {"contiguous": lambda a: a, "permuted": lambda a: [_permuted(t) if t.shape[2] > 6 else t for t in a],
         "padded": lambda a: [_padded(t) if i in (0, 4, 7) else t for i, t in enumerate(a)],
         "odd strides": lambda a: [_odd(t) if i in (0, 4) else t for i, t in enumerate(a)],
         "rows of a batch": lambda a: [t[1:] if t.shape[0] > 1 else t for t in a],
         "small tensors strided": lambda a: [_padded(t) if i in (1, 5, 6) else t for i, t in enumerate(a)]}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
def test_operator_is_the_same_through_both_paths(cuda, monkeypatch, dtype, form):
    a = FORMS[form](_operands(cuda, dtype))
    d_o = torch.randn(a[0].shape, generator=torch.Generator().manual_seed(1)).to(cuda, dtype)

    def everything():
        with torch.no_grad():
            plain = attentions.flashmvpa(*a, True, 0.125, window_size=2)
        leaves = [t.detach().requires_grad_() for t in a]
        o = attentions.flashmvpa(*leaves, True, 0.125, window_size=2)
        return [plain, o.detach(), *torch.autograd.grad(o, leaves, d_o)]

    native = everything()
    monkeypatch.setattr(mvpa_host, "usable", lambda t: False)
    for x, y in zip(native, everything()):
        assert x.shape == y.shape and x.stride() == y.stride() and torch.equal(x, y)


@pytest.mark.parametrize("change", [lambda a: a.__setitem__(4, torch.cat([a[4].flatten()[:1], a[4].flatten()])[1:].view(a[4].shape)),
                                    lambda a: a.__setitem__(0, a[0][:, :3]), lambda a: a.__setitem__(5, a[5][:, :, :4]),
                                    lambda a: a.__setitem__(1, a[1][..., :32]), lambda a: a.__setitem__(7, a[7][..., :32])])
def test_refused_calls_stay_refused(cuda, change):
    a = _operands(cuda, torch.bfloat16)
    change(a)
    with pytest.raises((AssertionError, RuntimeError)):
        attentions.flashmvpa(*a, True, 0.125, window_size=10)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_fused_branches_are_the_same_through_both_paths(cuda, monkeypatch, dtype):
    torch.manual_seed(0)
    block = MVPFormerBlock(models.MVPFormerConfig(n_embd=256, n_layer=1, n_head=4, n_head_kv=2, n_inner=320)).to(cuda, dtype).eval()
    B, T, C = 2, 14, 9
    x = torch.randn(B * T * C, 256, device=cuda).to(dtype)
    rt, rc = torch.randn(2, T, 64, device=cuda).to(dtype), torch.randn(2, C, 64, device=cuda).to(dtype)
    native = block.fused_branches(x, rt, rc, B, T, C)
    monkeypatch.setattr(mvpa_host, "usable", lambda t: False)
    assert torch.equal(native, block.fused_branches(x, rt, rc, B, T, C))
