"""GPU: relative keys that mask time steps out, with minus infinity or the type's lowest value in a feature that the queries hold at
one: no pair of the steps outside the content window counts, or none of the farthest ones, and the result is finite."""
import pytest
import torch

import attentions
import mvpa_port_torch as mp

pytestmark = pytest.mark.gpu


# the two forwards at head_dim 64 (many CTAs / few), 128 channel slots, head_dim 128, the CUDA-core kernel
@pytest.mark.parametrize("dtype, shape", [(torch.bfloat16, (1, 48, 12, 41, 24, 64)), (torch.bfloat16, (1, 48, 12, 41, 40, 64)),
                                          (torch.bfloat16, (1, 2, 1, 41, 24, 64)), (torch.bfloat16, (1, 2, 1, 41, 40, 64)),
                                          (torch.bfloat16, (1, 2, 1, 26, 70, 64)), (torch.bfloat16, (1, 2, 1, 41, 24, 128)),
                                          (torch.float32, (1, 2, 1, 41, 12, 64))])
@pytest.mark.parametrize("farther", [10, 13, 20])
@pytest.mark.parametrize("lowest", [False, True])
def test_masked_time_steps(cuda, dtype, shape, farther, lowest):
    B, H, Hkv, T, C, D = shape
    gen = torch.Generator().manual_seed(T * C + farther)
    r = lambda *s, std=1.0: (torch.randn(*s, D, generator=gen) * std).to(dtype)
    a = [r(B, H, T * C), r(1, Hkv, 1, std=0.1), r(1, Hkv, 1, std=0.1), r(1, Hkv, 1, std=0.1), r(B, Hkv, T * C), r(1, Hkv, T, std=0.3),
         r(1, Hkv, C, std=0.3), r(B, Hkv, T * C)]
    a[0][..., 0] = a[2][..., 0] = 1
    a[4][..., 0] = a[6][..., 0] = 0
    a[5][:, :, :T - 1 - farther, 0] = torch.finfo(dtype).min if lowest else -torch.inf      # slot T - 1 - (t_i - t_k)
    a = [t.to(cuda) for t in a]
    o = attentions.flashmvpa(*a, True, D ** -0.5, window_size=10)
    for j in range(0, Hkv, 5):
        heads = slice(j * (H // Hkv), (j + 1) * (H // Hkv))
        ref = mp.rel_attn(*(t.double() for t in (a[0][:, heads], *(t[:, j:j + 1] for t in a[1:]))), D ** -0.5, 10)
        assert torch.isfinite(ref).all()
        assert (o[:, heads] - ref).abs().max().item() <= (2e-2 if dtype == torch.bfloat16 else 1e-5) * max(1.0, ref.abs().max().item())
