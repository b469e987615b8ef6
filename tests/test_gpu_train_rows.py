"""GPU: the differentiable RMSNorm and SwiGLU of the training path at the edges of their launch shapes, against torch in
64 bits, and the routes that torch expressions keep serving."""
import pytest
import torch

import mvpa_ops

pytestmark = pytest.mark.gpu

# fp32: sums of up to 4096 terms; bf16 (unit roundoff 2^-8): one rounding of the result around fp32 arithmetic, and for
# SwiGLU a second one, of silu(gate) before the product, as eager PyTorch does
TOL = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -8}
TOL_SWIGLU = {torch.float32: 2e-6, torch.bfloat16: 2 * 2.0 ** -8}


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
