"""GPU: which kernel a call takes, by the names that the profiler sees (equal results do not tell)."""
import re

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import attentions
import test_gpu_tiles

pytestmark = pytest.mark.gpu

TWO = next(m for m in test_gpu_tiles.test_two_ctas_per_multiprocessor_bf16.pytestmark if m.name == "parametrize").args[1]


def _kernels(call):
    with profile(activities=[ProfilerActivity.CUDA]) as prof, torch.no_grad():
        call()
        torch.cuda.synchronize()
    return [n for e in prof.events() for n in re.findall(r"\w+_kernel", e.name)]


def _call(cuda, B, H, Hkv, T, C, D, window=10, q_time=None):
    r = lambda *s: torch.randn(*s, D, device=cuda).bfloat16()
    q = r(B, H, (T if q_time is None else q_time[1]) * C)
    return _kernels(lambda: attentions.flashmvpa(q, r(1, Hkv, 1), r(1, Hkv, 1), r(1, Hkv, 1), r(B, Hkv, T * C), r(1, Hkv, T), r(1, Hkv, C),
                                                 r(B, Hkv, T * C), True, D ** -0.5, window_size=window, q_time_range=q_time))


# the cases that compare the two forwards at head_dim 64 do run both: two CTAs per multiprocessor for the whole call where its
# window leaves at most sixteen dense key steps beside light tiles, the other kernel for one kv head alone
@pytest.mark.parametrize("shape, window, q_time", TWO)
def test_both_forwards_of_a_comparison(cuda, shape, window, q_time):
    B, H, Hkv, T, C = shape
    steps = 4 if C <= 32 else 2                      # key steps of a tile
    tiles = -(-T // steps)
    light = window > 0 and tiles >= 2 and (tiles - 2) * steps - steps - window >= 0
    fits = not light or (-(-window // steps) + 1) * steps <= 16
    whole = _call(cuda, B, H, Hkv, T, C, 64, window, q_time)
    assert ("tc_fwd_two_kernel" in whole) == fits and ("tc_fwd_kernel" in whole) != fits
    if B * Hkv > 1:
        alone = _call(cuda, 1, H // Hkv, 1, T, C, 64, window, q_time)
        assert "tc_fwd_kernel" in alone and "tc_fwd_two_kernel" not in alone


def test_pre_kernel(cuda):
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert _call(cuda, 1, sms, sms, 1, 100, 128).count("rel_const_kernel") == 0        # every CTA resident at once
    assert _call(cuda, 1, sms + 1, sms + 1, 1, 100, 128).count("rel_const_kernel") == 1
