"""GPU: which calls the native host path takes, asked of it directly (what it declines goes through Python, with the same
result, which a comparison of results does not show)."""
import pytest
import torch

import attentions
import models
import mvpa_host
from test_gpu_host_path import FORMS, _operands

pytestmark = pytest.mark.gpu


def _attend(a):
    return mvpa_host.module().attend(*a, 0.125, 2, False)


def _record(a):
    return mvpa_host.module().forward(*a, 0.125, 2, 0, 0, False)


def _grads(a, d_o, record):
    return mvpa_host.module().backward(d_o, *a, *record, 0.125, 2, False)


# layouts that the kernels read in place are taken; what has to be copied first is not
@pytest.mark.parametrize("form, taken", [("contiguous", True), ("permuted", True), ("padded", True), ("rows of a batch", True),
                                         ("odd strides", False), ("small tensors strided", False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
def test_operator_forms(cuda, dtype, form, taken):
    with torch.no_grad():
        a = FORMS[form](_operands(cuda, dtype))
        assert mvpa_host.usable(a[0]) and (_attend(a) is not None) == taken
        record = _record(a)
        assert (record is not None) == taken
        if taken:
            assert _grads(a, torch.ones_like(a[0]), record) is not None
            assert _grads(a, torch.ones_like(a[0])[..., ::2].repeat_interleave(2, -1).transpose(2, 3).contiguous().transpose(2, 3), record) is not None


def test_operator_calls_that_python_has_to_see(cuda):
    a = _operands(cuda, torch.bfloat16)
    assert _attend([a[0].clone().requires_grad_(), *a[1:]]) is None            # a gradient flows
    assert _attend([*a[:5], a[5].float(), *a[6:]]) is None                     # another type
    assert _attend([*a[:7], a[7].cpu()]) is None
    assert _attend([a[0], *a[1:4], a[4][:1], *a[5:7], a[7][:1]]) is None       # another batch
    assert mvpa_host.module().attend(*a, 1, 2, False) is None                  # a scale that is no float


class _Functions(torch.overrides.TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


# a default device watches nothing; a mode that sees each call, alone or under one, does
def test_default_device(cuda):
    a = _operands(cuda, torch.bfloat16)
    block = models.MVPFormerBlock(models.MVPFormerConfig(n_embd=256, n_layer=1, n_head=4, n_head_kv=2, n_inner=320)).to(cuda).eval()
    w_in, w_out = block.fused_weights()
    r = lambda *s: torch.randn(*s, device=cuda)
    x, rt, rc, bias = r(2 * 30, 256), r(2, 5, 64), r(2, 6, 64), block.attn.attn_bias.detach()

    def taken():
        return [_attend(a) is not None, _record(a) is not None, mvpa_host.module().plain(a[0], a[4]) == 1,
                mvpa_host.module().branches(x, w_in, w_out, bias, rt, rc, 10, 2, 5, 6, 4, 2, 64, False) is not None]

    assert all(taken())
    for device in (cuda, "cpu"):
        with torch.device(device):
            assert all(taken())
            with _Functions():
                assert not any(taken())
        with _Functions(), torch.device(device):
            assert not any(taken())


# operands that do not go together are refused before a kernel reads them, on every way to the kernels
@pytest.mark.parametrize("change", [lambda a: (4, a[4][:1]), lambda a: (7, a[7][:1]), lambda a: (7, a[7][:, :, :-1]), lambda a: (4, a[4][:, :1]),
                                    lambda a: (4, a[4].float()), lambda a: (1, a[1].float()), lambda a: (5, a[5].half()), lambda a: (7, a[7].cpu()),
                                    lambda a: (2, a[2].cpu())])
@pytest.mark.parametrize("grad", [False, True])
def test_operands_that_do_not_go_together(cuda, change, grad):
    a = _operands(cuda, torch.bfloat16)
    i, t = change(a)
    a[i] = t
    if grad:
        a[0].requires_grad_()
    with pytest.raises((RuntimeError, AssertionError)):
        attentions.flashmvpa(*a, True, 0.125, window_size=10)
    small = [x[0] if j in (1, 2, 3, 5, 6) else x for j, x in enumerate(a)]
    with pytest.raises((RuntimeError, AssertionError)), torch.no_grad():
        attentions.flash_mvpa_into(torch.empty_like(a[0]), *small, 0.125, 10)


def test_output_of_another_type(cuda):
    a = _operands(cuda, torch.bfloat16)
    small = [x[0] if j in (1, 2, 3, 5, 6) else x for j, x in enumerate(a)]
    with pytest.raises(RuntimeError):
        attentions.flash_mvpa_into(torch.empty_like(a[0], dtype=torch.float32), *small, 0.125, 10)


# saved tensors that a hook brings back in another layout, on both ways to the kernels
@pytest.mark.parametrize("form", [lambda t: t.clone(), lambda t: torch.nn.functional.pad(t, (0, 1))[..., :-1],
                                  lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_backward_of_rearranged_saved_tensors(cuda, dtype, form):
    a = [t.requires_grad_() for t in _operands(cuda, dtype)]
    d_o = torch.ones_like(a[0])
    want = torch.autograd.grad(attentions.flashmvpa(*a, True, 0.125, window_size=2), a, d_o)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), form):
        o = attentions.flashmvpa(*a, True, 0.125, window_size=2)
    for g, w in zip(torch.autograd.grad(o, a, d_o), want):
        assert torch.equal(g, w)
