"""CPU: host-side logic of the model-level package: state-dict layout against the fixture written from the
reference's `MVPFormerModel`, configuration aliases, encoder sizes, and the synthetic iEEG generator."""
import numpy as np
import torch

import models
from eeg_datasets import synthetic_ieeg
from models import block_grad
from test_model_oracle import load_model_golden


def _config(cfg, **kw):
    return models.MVPFormerConfig(n_positions=cfg["n_positions"], n_channels=cfg["n_channels"], n_embd=cfg["n_embd"],
                                  n_layer=cfg["n_layer"], n_head=cfg["n_head"], n_inner=cfg["n_inner"],
                                  n_head_kv=cfg["n_head_kv"], layer_norm_epsilon=cfg["eps"], **kw)


def test_state_dict_has_the_reference_keys_and_shapes():
    g, cfg, state = load_model_golden()
    m = models.MVPFormerModel(_config(cfg))
    own = {k: v for k, v in m.state_dict().items() if not k.endswith(("time_bias", "masked_bias"))}
    assert set(own) == set(state)
    for k, v in own.items():
        assert tuple(v.shape) == tuple(state[k].shape), k
    m.load_state_dict(state, strict=False)             # the two buffers are not in the fixture
    assert torch.equal(m.h[1].mlp.up_proj.weight, state["h.1.mlp.up_proj.weight"])


def test_config_aliases_and_task_layout():
    c = models.MVPFormerConfig(n_embd=768, n_layer=12, n_head=12, n_head_kv=4, n_inner=1728, n_positions=128)
    assert (c.hidden_size, c.num_attention_heads, c.num_hidden_layers, c.intermediate_size) == (768, 12, 12, 1728)
    assert c.max_position_embeddings == 128 and c.max_channel_embeddings == 128
    enc = models.WaveEncoder(2560, 768)
    assert enc.dwt_size == 2610 and enc.sizes == [1283, 645, 326, 166, 86, 46, 26, 16, 16]
    task = models.ClassificationHMVPFormer(models.MVPFormerConfig(n_embd=64, n_layer=1, n_head=4, n_head_kv=2, n_inner=96),
                                           models.WaveEncoder(256, 64), models.MVPFormerHead(64, 2))
    keys = set(task.state_dict())
    assert {"seizure_embeddings", "encoder.ln.weight", "encoder.proj.weight", "head.head.weight",
            "mvpformer.ln_f.weight", "mvpformer.h.0.attn.attn_bias", "mvpformer.h.0.mlp.down_proj.weight"} <= keys


def test_negative_indices_never_name_the_token_itself():
    task = models.HMVPFormer(models.MVPFormerConfig(n_embd=64, n_layer=1, n_head=4, n_head_kv=2, n_inner=96),
                             models.WaveEncoder(256, 64), models.MVPFormerHead(64), num_negatives=7)
    idx = task._negative_indices((3, 5, 4), torch.Generator().manual_seed(0))
    n = 3 * 5 * 4
    assert idx.shape == (3, 5, 4, 7) and idx.dtype == torch.int32
    assert int(idx.min()) >= 0 and int(idx.max()) < n
    own = torch.arange(n).view(3, 5, 4, 1)
    assert not (idx == own).any()


def test_synthetic_ieeg_is_seeded_pink_and_bursty():
    a = synthetic_ieeg(1, 16, 4, 512, seed=3)
    b = synthetic_ieeg(1, 16, 4, 512, seed=3)
    assert a.shape == (1, 16, 4, 512) and a.dtype == torch.float32 and torch.equal(a, b)
    assert not torch.equal(a, synthetic_ieeg(1, 16, 4, 512, seed=4))
    quiet = synthetic_ieeg(1, 16, 4, 512, seed=3, bursts=0)
    rec = quiet[0].permute(1, 0, 2).reshape(4, -1).double()                     # (channels, time)
    assert abs(float(rec.mean())) < 1e-3 and abs(float(rec.std()) - 1.0) < 1e-2  # z-scored per channel
    p = np.abs(np.fft.rfft(rec.numpy(), axis=-1)) ** 2
    f = np.fft.rfftfreq(rec.shape[-1], d=1 / 512.0)
    lo, hi = (f > 1) & (f < 4), (f > 64) & (f < 256)
    slope = np.log(p[:, hi].mean() / p[:, lo].mean()) / np.log(f[hi].mean() / f[lo].mean())
    assert -1.3 < slope < -0.7                                                   # power ~ 1/f
    assert float(a.abs().max()) > 4.0 > float(quiet.abs().max()) * 0.8           # bursts stand out of the background


class _Step(torch.autograd.Function):
    """A block whose backward always goes through the differentiable expression: x + tanh(x * e) * w."""
    calls = 0

    @staticmethod
    def f(x, e, w):
        return x + torch.tanh(x * e) * w

    @staticmethod
    def forward(ctx, x, e, w):
        ctx.save_for_backward(x, e, w)
        return _Step.f(x, e, w)

    @staticmethod
    def backward(ctx, dy):
        _Step.calls += 1
        return tuple(block_grad.through_expression(_Step.f, ctx.saved_tensors, ctx.needs_input_grad, dy))


def test_gradients_through_the_expression_stop_at_the_block():
    """Stacked blocks that share a non-leaf input: first and second derivatives, one backward call per block."""
    g = torch.Generator().manual_seed(0)
    x, w, a = (torch.randn(3, dtype=torch.float64, generator=g, requires_grad=True) for _ in range(3))
    ins, dy = (x, w, a), torch.randn(3, dtype=torch.float64, generator=g)

    def run(step):
        e, y = a * 2, x
        for _ in range(6):
            y = step(y, e, w)
        first = torch.autograd.grad(y, ins, dy, create_graph=True)
        return first, torch.autograd.grad(sum((t * t).sum() for t in first), ins)

    _Step.calls = 0
    plain = torch.autograd.grad(_Step.apply(x, a * 2, w), ins, dy)
    assert _Step.calls == 1 and not any(t.requires_grad for t in plain)
    _Step.calls = 0
    got = run(_Step.apply)
    assert _Step.calls <= 6 + 6          # (the second derivative may run each block's graph, never the blocks below it)
    for p, q in zip(got, run(_Step.f)):
        for s, t in zip(p, q):
            torch.testing.assert_close(s, t, rtol=1e-12, atol=1e-12)


def test_mlp_can_be_traced_scripted_and_compiled():
    m = models.mvpformer.LlamaMLP(models.MVPFormerConfig(n_embd=8, n_inner=16))
    x = torch.randn(3, 8)
    want = m.down_proj(torch.nn.functional.silu(m.gate_proj(x)) * m.up_proj(x))
    for form in (m, torch.fx.symbolic_trace(m), torch.jit.script(m), torch.jit.trace(m, x),
                 torch.compile(m, backend="eager", fullgraph=True), torch.export.export(m, (x,)).module(), torch.vmap(m)):
        torch.testing.assert_close(form(x), want)


def test_the_fused_gate_starts_at_its_size(monkeypatch):
    calls = []
    monkeypatch.setattr(models.mvpformer.mvpa_ops, "swiglu",
                        lambda g, u: calls.append(g.shape) or torch.nn.functional.silu(g) * u)
    m = models.mvpformer.LlamaMLP(models.MVPFormerConfig(n_embd=8, n_inner=16))
    m(torch.randn(300, 8))
    assert not calls                                   # far below the line: torch's two launches
    monkeypatch.setattr(models.mvpformer, "GATE_BYTES", 300 * 16 * 4)
    m(torch.randn(299, 8))
    m(torch.randn(300, 8))
    assert calls == [(300, 16)]


def test_scratch_sizes_are_asked_for_on_the_tensors_device(monkeypatch):
    """The norm's backward sizes its scratch by the multiprocessors of the current device: that has to be x's."""
    from contextlib import contextmanager
    import mvpa_ops
    current, asked = ["another"], []

    @contextmanager
    def on_device(device):
        current.append(device)
        yield
        current.pop()

    class Lib:
        def mvpa_rmsnorm_bwd_workspace_bytes(self, rows, width):
            asked.append(current[-1])
            return 16

        def mvpa_rmsnorm_bwd(self, *args):
            asked.append(current[-1])
            return 0

    monkeypatch.setattr(mvpa_ops._nat, "lib", Lib)
    monkeypatch.setattr(mvpa_ops._nat, "on_device", on_device)
    monkeypatch.setattr(mvpa_ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(mvpa_ops, "_stream", lambda t: None)
    x = torch.zeros(3, 8)
    mvpa_ops.rmsnorm_bwd(x, x[0], x, 1e-5)
    assert asked == [x.device, x.device]
