"""GPU: calls that follow each other without a pause, each reading what the one before wrote.  (Everywhere else the kernels' status is
read back after each call, which waits for it: launches that come up while the kernel before them runs out do not overlap there.)"""
import pytest
import torch

import attentions
import mvpa_ops
from attentions import attn

pytestmark = pytest.mark.gpu

# two sizes in turn: no pre-kernel / more CTAs than multiprocessors, one and two CTAs per multiprocessor, CUDA cores
PAIRS = {"small 64": (torch.bfloat16, (1, 12, 4, 6, 22, 64), (1, 12, 4, 3, 17, 64)),
         "small and large 64": (torch.bfloat16, (1, 4, 2, 5, 30, 64), (2, 24, 8, 25, 33, 64)),
         "small and large 128": (torch.bfloat16, (1, 8, 4, 6, 22, 128), (1, 16, 8, 25, 100, 128)),
         "small 64 and 128 channels": (torch.bfloat16, (1, 4, 4, 12, 40, 64), (1, 6, 2, 7, 100, 64)),
         "fp32": (torch.float32, (1, 4, 2, 12, 22, 64), (1, 2, 1, 9, 8, 32))}


def _case(cuda, dtype, shape):
    B, H, Hkv, T, C, D = shape
    gen = torch.Generator().manual_seed(sum(shape))
    r = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(cuda, dtype)
    return [r(B, H, T * C, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(1, Hkv, 1, D), r(B, Hkv, T * C, D), r(1, Hkv, T, D, std=0.3),
            r(1, Hkv, C, D, std=0.3), r(B, Hkv, T * C, D)], r(B, H, T * C, D)


def _forward(a, q):
    return attentions.flashmvpa(q, *a[1:], True, a[0].shape[-1] ** -0.5, window_size=10)


def _norm(q):          # the row kernels between two operators
    D = q.shape[-1]
    rows = q.contiguous().view(-1, D)
    y = mvpa_ops.rmsnorm(rows, torch.ones(D, device=q.device, dtype=q.dtype), 1e-5)
    return mvpa_ops.silu_mul(y, y, torch.empty_like(y)).view(q.shape)


def _chain(cases, count, between):
    """`count` forwards of the cases in turn, each on what its case's last one gave."""
    qs, outs = [a[0] for a, _ in cases], []
    with torch.no_grad():
        for i in range(count):
            j = i % len(cases)
            qs[j] = _norm(_forward(cases[j][0], qs[j]))
            outs.append(qs[j])
            between()
    return outs


@pytest.mark.parametrize("pair", PAIRS)
def test_forwards(cuda, monkeypatch, pair):
    monkeypatch.setattr(attn, "_CHECK_STATUS", False)
    dtype, *shapes = PAIRS[pair]
    cases = [_case(cuda, dtype, s) for s in shapes]
    want = _chain(cases, 120, torch.cuda.synchronize)
    for got, w in zip(_chain(cases, 120, lambda: None), want):
        assert torch.equal(got, w)


@pytest.mark.parametrize("pair", PAIRS)
def test_forwards_and_backwards(cuda, monkeypatch, pair):
    monkeypatch.setattr(attn, "_CHECK_STATUS", False)
    dtype, *shapes = PAIRS[pair]
    cases = [_case(cuda, dtype, s) for s in shapes]

    def steps(between):
        outs, dos = [], [do for _, do in cases]
        for i in range(40):
            j = i % len(cases)
            leaves = [t.detach().requires_grad_() for t in cases[j][0]]
            o = _forward(leaves, leaves[0])
            between()
            grads = torch.autograd.grad(o, leaves, dos[j])
            between()
            dos[j] = _norm(grads[0])                 # the next backward reads what this one wrote
            outs += [o.detach(), *grads]
        return outs

    want = steps(torch.cuda.synchronize)
    for got, w in zip(steps(lambda: None), want):
        assert torch.equal(got, w)


# the same captured in a graph, with a stream beside it whose work joins in between
@pytest.mark.parametrize("pair", PAIRS)
def test_captured_with_a_side_stream(cuda, monkeypatch, pair):
    monkeypatch.setattr(attn, "_CHECK_STATUS", False)
    dtype, *shapes = PAIRS[pair]
    cases = [_case(cuda, dtype, s) for s in shapes]
    side = torch.cuda.Stream()

    def work(overlap):
        outs, (a, q), (a2, q2) = [], (cases[0][0], cases[0][0][0]), (cases[1][0], cases[1][0][0])
        with torch.no_grad():
            for _ in range(8):
                main = torch.cuda.current_stream()
                side.wait_stream(main) if overlap else None
                with torch.cuda.stream(side if overlap else main):
                    q2 = _norm(_forward(a2, q2))
                q = _norm(_forward(a, q))
                main.wait_stream(side) if overlap else None
                outs += [q + q2.mean(), _norm(q2)]   # (and a row kernel that reads what the other stream wrote)
                q2 = outs[-1]
        return outs

    want = [t.clone() for t in work(False)]
    warm = torch.cuda.Stream()
    warm.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(warm):
        work(True)
    torch.cuda.current_stream().wait_stream(warm)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = work(True)
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        for got, w in zip(outs, want):
            assert torch.equal(got, w)
