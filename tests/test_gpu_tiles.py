"""GPU: the tiled CUDA-core kernels and the training kernels of the block at the edges of their tiles and on both
sides of each launch rule, against the oracle (operator) and torch in 64 bits (row kernels)."""
import numpy as np
import pytest
import torch

import attentions
import mvpa_oracle as mo
import mvpa_port_torch as mp
from test_gpu_op import BF16_ABS, F16_ABS, F32_REL, GRADS, _np, _op, _oracle_args, _rounded, random_case

pytestmark = pytest.mark.gpu

TOL = {torch.float32: F32_REL, torch.float16: F16_ABS, torch.bfloat16: BF16_ABS}


def _check(cuda, g, dtype, window=10):
    """Forward and all eight gradients against the oracle at the operator tests' tolerances."""
    gr = g if dtype == torch.float32 else _rounded(g, dtype)
    o, t = _op(cuda, g, dtype, grads=True, window=window)
    o.backward(torch.tensor(g["do"], device=cuda, dtype=dtype))
    ref_o = mo.mvpa_forward(*_oracle_args(gr), float(g["sm_scale"]), window=window)[0]
    ref = mo.mvpa_backward(*_oracle_args(gr), gr["do"], float(g["sm_scale"]), window=window)
    pairs = [("o", o, ref_o)] + [(n, t[k].grad, ref[n]) for n, k in zip(
        GRADS, ("q", "u", "v", "z", "k", "r_time", "r_chan", "val"))]
    for name, got, want in pairs:
        err = np.abs(_np(got).reshape(np.shape(want)) - want).max()
        assert err <= TOL[dtype] * max(1.0, np.abs(want).max()), (name, err)


# (B, H, Hkv, T, C, D): fewer rows than a tile, one row and one key past a tile, ragged channels that put a time
# step's end inside a tile, light tiles (T > window + tile), and every head_dim
@pytest.mark.parametrize("shape", [(1, 2, 1, 1, 3, 64), (1, 2, 1, 1, 17, 16), (2, 4, 2, 5, 13, 64), (1, 2, 2, 3, 43, 32),
                                   (1, 2, 1, 24, 11, 128), (1, 1, 1, 45, 3, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_cuda_core_tiles_sixteen_rows(cuda, shape, dtype):
    _check(cuda, random_case(sum(shape), *shape), dtype)


# more sixteen-row tiles than four per multiprocessor: thirty-two rows per CTA, last tile ragged; at D 64 and 128 light
# tiles too (T > window + tile), and at the last two the key side stays below the line, with query heads above it
@pytest.mark.parametrize("shape", [(2, 16, 16, 15, 21, 16), (1, 32, 16, 17, 19, 32), (2, 16, 16, 24, 13, 64), (2, 16, 16, 24, 13, 128),
                                   (1, 64, 8, 24, 13, 64), (1, 64, 8, 24, 13, 128)])
def test_cuda_core_tiles_thirty_two_rows(cuda, shape):
    _check(cuda, random_case(sum(shape), *shape), torch.float32)


# key side in clusters of two CTAs: an odd number of items, the last of a ragged tile, one item more than a CTA's groups, light
# items, two heads a group, and each head_dim
@pytest.mark.parametrize("shape", [(1, 2, 1, 9, 17, 16), (1, 5, 1, 5, 12, 32), (1, 4, 2, 24, 11, 64), (1, 1, 1, 45, 11, 64), (2, 2, 1, 13, 17, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_cuda_core_key_side_in_pairs(cuda, shape, dtype):
    _check(cuda, random_case(sum(shape), *shape), dtype)


# time / channel axes whose slot sums do not fit beside the four groups' tiles
@pytest.mark.parametrize("shape", [(1, 1, 1, 2, 400, 64), (1, 1, 1, 300, 2, 128), (1, 2, 1, 2, 440, 32)])
def test_cuda_core_long_axes(cuda, shape):
    _check(cuda, random_case(sum(shape), *shape), torch.float32)


# key-side tensor-core pipeline: one, two and three dense pairs, then the first light pairs, one and two heads a
# group, both head_dims and each number of channel slots
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 100, 128), (1, 2, 1, 2, 128, 128), (1, 1, 1, 3, 70, 128), (1, 2, 1, 13, 65, 128),
                                   (1, 2, 1, 27, 33, 128), (1, 1, 1, 45, 20, 128), (1, 1, 1, 2, 100, 64), (1, 2, 1, 14, 100, 64),
                                   (1, 2, 1, 27, 50, 64), (1, 1, 1, 49, 32, 64)])
def test_key_side_pipeline_bf16(cuda, shape):
    _check(cuda, random_case(sum(shape), *shape, scale=0.5), torch.bfloat16)


# two CTAs per multiprocessor (head_dim 64, at most 64 channel slots, more CTAs than multiprocessors): one and several time
# steps, the last tile's scores all in tensor memory (T <= 64) and half of them in shared memory, the first light tile, each
# number of channel slots, windows with no, few and the most dense key steps beside light tiles and one more, a query range
@pytest.mark.parametrize("shape, window, q_time", [
    ((1, 180, 90, 1, 22), 10, None), ((2, 48, 8, 7, 32), 10, None), ((1, 52, 13, 16, 31), 10, None), ((1, 28, 7, 17, 64), 10, None),
    ((1, 14, 7, 64, 33), 10, None), ((1, 14, 14, 65, 40), 10, None), ((1, 14, 2, 128, 17), 10, None), ((1, 11, 1, 128, 34), 10, None),
    ((1, 16, 4, 100, 16), 0, None), ((1, 16, 4, 100, 16), 1, None), ((1, 16, 4, 100, 16), 12, None), ((1, 16, 4, 100, 16), 13, None),
    ((1, 12, 4, 77, 36), 14, None), ((1, 12, 4, 77, 36), 15, None), ((1, 12, 4, 77, 36), 80, None), ((2, 18, 6, 90, 20), 10, (28, 40))])
def test_two_ctas_per_multiprocessor_bf16(cuda, shape, window, q_time):
    B, H, Hkv, T, C = shape
    gen = torch.Generator().manual_seed(sum(shape) + window)
    r = lambda *s: torch.randn(*s, 64, generator=gen).to(cuda, torch.bfloat16)
    a = [r(B, H, T * C), r(1, Hkv, 1), r(1, Hkv, 1), r(1, Hkv, 1), r(B, Hkv, T * C), r(1, Hkv, T), r(1, Hkv, C), r(B, Hkv, T * C)]
    rows = slice(None) if q_time is None else slice(q_time[0] * C, sum(q_time) * C)
    o = attentions.flashmvpa(a[0][:, :, rows].contiguous(), *a[1:], True, 0.125, window_size=window, q_time_range=q_time)
    for b in range(B):
        for j in range(Hkv):       # (one kv head at a time: the reference materialises its scores)
            heads = slice(j * (H // Hkv), (j + 1) * (H // Hkv))
            per = [a[0][b:b + 1, heads], *(t[:, j:j + 1] for t in a[1:4]), a[4][b:b + 1, j:j + 1], *(t[:, j:j + 1] for t in a[5:7]),
                   a[7][b:b + 1, j:j + 1]]
            ref = mp.rel_attn(*(t.double() for t in per), 0.125, window if window > 0 else T)[:, :, rows]
            got = o[b:b + 1, heads]
            assert (got - ref).abs().max().item() <= BF16_ABS * max(1.0, ref.abs().max().item())
            # one kv head's call is too small for this kernel: the other one, the same bits
            alone = attentions.flashmvpa(per[0][:, :, rows].contiguous(), *(t.contiguous() for t in per[1:]), True, 0.125,
                                         window_size=window, q_time_range=q_time)
            assert torch.equal(got, alone)


@pytest.mark.parametrize("shape", [(1, 52, 13, 14, 18, 64), (2, 24, 12, 9, 37, 64)])
def test_two_ctas_per_multiprocessor_backward_of_its_forward(cuda, shape):
    _check(cuda, random_case(sum(shape), *shape, scale=0.5), torch.bfloat16)


# fp32 sums at the smallest sizes, where the score products' rounding is all there is: root mean square over fifty draws of
# the relative error against 64 bits.  A product of 64 terms in four chains measures 1.14e-7 (output) and 2.24e-7 (dq), in
# groups of four terms 1.21e-7 and 2.28e-7, in two chains 1.28e-7 and 2.49e-7: the limits lie above the second.
def test_fp32_scores_round_no_more_than_a_sum_in_groups(cuda):
    B, H, Hkv, T, C, D = 1, 2, 1, 4, 4, 64
    errors = []
    for seed in range(50):
        gen = torch.Generator().manual_seed(seed)
        r = lambda *s, std=1.0: (torch.randn(*s, generator=gen) * std).to(cuda)
        a = [r(B, H, T * C, D), r(1, Hkv, 1, D, std=0.1), r(1, Hkv, 1, D, std=0.1), r(1, Hkv, 1, D, std=0.1), r(B, Hkv, T * C, D),
             r(1, Hkv, T, D, std=0.3), r(1, Hkv, C, D, std=0.3), r(B, Hkv, T * C, D)]
        do = r(B, H, T * C, D)
        q = a[0].requires_grad_()
        o = attentions.flashmvpa(*a, True, D ** -0.5, window_size=10)
        q64 = q.detach().double().requires_grad_()
        o64 = mp.rel_attn(q64, *(t.double() for t in a[1:]), D ** -0.5, 10)
        pairs = (o, o64), (torch.autograd.grad(o, q, do)[0], torch.autograd.grad(o64, q64, do.double())[0])
        errors.append([((x.double() - y).norm() / y.norm()).item() ** 2 for x, y in pairs])
    rms_o, rms_dq = np.sqrt(np.mean(errors, axis=0))
    assert rms_o <= 1.23e-7 and rms_dq <= 2.33e-7
