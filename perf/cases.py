"""The work that users of this package have it do, as measurable cases: the operator on its own (inference and training,
bf16 and fp32), whole-model inference on raw iEEG (one live window, a batch, the long-context next-state task) and a training
step of the block stack.  Every case goes through the public entry points: `attentions.flashmvpa`, `models.*`.

Sizes come from the shipped configurations (MVPFormer-S: width 768, 12 layers, 12 heads over 4 kv heads of 64; the generative
model: width 2048, 24 layers, 16 heads over 8 kv heads of 128; segments of 2560 samples, loader windows of 25 segments, up to
128 segments, patients with 22 to 128 channels), from the benchmark's workloads and from the tests.
"""
from __future__ import annotations

import importlib
import math

import torch

importlib.import_module("multi-variate-parallel-transformer_b200")  # puts the package's folders on sys.path

import attentions  # noqa: E402
import models  # noqa: E402
from eeg_datasets import synthetic_ieeg  # noqa: E402

WINDOW = 10          # content window of every shipped configuration
SEGMENT = 2560       # samples of a five-second segment at 512 Hz
NEGATIVES = 30       # sampled negatives of the next-state task
ARCH = {
    "s": dict(n_embd=768, n_layer=12, n_head=12, n_head_kv=4, n_inner=1728),
    "generative": dict(n_embd=2048, n_layer=24, n_head=16, n_head_kv=8, n_inner=5632),
}
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def listed():
    return [
        # the operator alone, forward: a six-segment window of a 22-channel patient (latency and launches)
        dict(name="attend_small", kind="attend", dtype="bf16", B=1, H=12, Hkv=4, T=6, C=22, D=64),
        # the benchmark's fp32 configuration: 16 channels x 32 segments, exact fp32 arithmetic
        dict(name="attend_fp32", kind="attend", dtype="fp32", B=1, H=4, Hkv=4, T=32, C=16, D=64),
        # the benchmark's headline workload: 4096 tokens, head_dim 64
        dict(name="attend_4k", kind="attend", dtype="bf16", B=4, H=16, Hkv=16, T=64, C=64, D=64),
        # long context: 128 channels x 128 segments, one attention layer of the generative model
        dict(name="attend_16k", kind="attend", dtype="bf16", B=1, H=16, Hkv=8, T=128, C=128, D=128),
        # forward + backward in fp32 at a test's size: gradient checks, fine-tuning in full precision
        dict(name="train_fp32", kind="attend_train", dtype="fp32", B=1, H=4, Hkv=2, T=24, C=22, D=64),
        # forward + backward at the loader's window of 25 segments, a ragged channel count, the generative model's heads
        dict(name="train_ragged", kind="attend_train", dtype="bf16", B=4, H=16, Hkv=8, T=25, C=100, D=128),
        # the benchmark's training configuration: 32 channels x 128 segments, head_dim 64
        dict(name="train_4k", kind="attend_train", dtype="bf16", B=8, H=16, Hkv=16, T=128, C=32, D=64),
        # the same at long context
        dict(name="train_16k", kind="attend_train", dtype="bf16", B=1, H=16, Hkv=8, T=128, C=128, D=128),
        # one live window of one patient through the small model (monitoring: frozen weights, CUDA graph)
        dict(name="classify_one", kind="classify", arch="s", B=1, T=25, C=22, graph=True),
        # seizure classification of a batch of long recordings, the benchmark's fourth configuration
        dict(name="classify_batch", kind="classify", arch="s", B=8, T=128, C=64, graph=False),
        # next-state logits of the generative model at long context (two samples of the benchmark's fifth configuration)
        dict(name="next_state", kind="next_state", arch="generative", B=2, T=128, C=128, graph=False),
        # one training step (forward, loss, backward) of the small model's block stack at the loader's window
        dict(name="train_model", kind="model_train", arch="s", B=4, T=25, C=64),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm; odd values come as they fall."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["attend", "attend", "attend_train", "attend_train", "classify", "next_state", "model_train"])
    if kind in ("attend", "attend_train"):
        if rng.random() < 0.2:
            D, Hkv = rng.choice([32, 64, 128]), rng.choice([1, 2, 4])
            return dict(kind=kind, dtype="fp32", B=rng.choice([1, 2]), H=Hkv * rng.choice([1, 2]), Hkv=Hkv, T=_log(rng, 4, 48),
                        C=_log(rng, 4, 32), D=D)
        H, Hkv, D = rng.choice([(12, 4, 64), (16, 16, 64), (16, 8, 128)])
        T, C = _log(rng, 3, 128), _log(rng, 16, 128)
        top = max(1, min(8, 65536 // (T * C)))
        return dict(kind=kind, dtype="bf16", B=_log(rng, 1, top), H=H, Hkv=Hkv, T=T, C=C, D=D)
    if kind == "classify":
        T, C = _log(rng, 8, 128), _log(rng, 16, 128)
        return dict(kind=kind, arch="s", B=_log(rng, 1, max(1, min(8, 65536 // (T * C)))), T=T, C=C, graph=rng.random() < 0.5)
    if kind == "next_state":
        T, C = _log(rng, 12, 128), _log(rng, 16, 128)
        return dict(kind=kind, arch="generative", B=_log(rng, 2, max(2, min(8, 32768 // (T * C)))), T=T, C=C,
                    graph=rng.random() < 0.5)
    T, C = _log(rng, 8, 64), _log(rng, 16, 128)
    return dict(kind=kind, arch="s", B=_log(rng, 1, max(1, min(8, 16384 // (T * C)))), T=T, C=C)


# ---------------------------------------------------------------------------------------------------------------------
def _config(arch):
    # dropout off: a pass is then a function of its inputs (the shipped rate only scales what the kernels produce)
    return models.MVPFormerConfig(n_positions=128, n_channels=128, resid_pdrop=0.0, embd_pdrop=0.0, attn_pdrop=0.0, **ARCH[arch])


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    kind = case["kind"]
    if kind in ("attend", "attend_train"):
        dt = DTYPES[case["dtype"]]
        B, H, Hkv, T, C, D = (case[k] for k in ("B", "H", "Hkv", "T", "C", "D"))
        N = T * C
        r = lambda *s, std=1.0: (torch.randn(*s, generator=gen, device=dev) * std).to(dt)
        # normalised projections; biases and relative keys of a partly trained layer
        args = [r(B, H, N, D), r(1, Hkv, 1, D, std=0.1), r(1, Hkv, 1, D, std=0.1), r(1, Hkv, 1, D, std=0.1), r(B, Hkv, N, D),
                r(1, Hkv, T, D, std=0.3), r(1, Hkv, C, D, std=0.3), r(B, Hkv, N, D)]
        state = dict(kind=kind, args=args, scale=D ** -0.5)
        if kind == "attend_train":
            for a in args:
                a.requires_grad_(True)
            state["d_o"] = r(B, H, N, D)
        return state
    B, T, C, arch = case["B"], case["T"], case["C"], case["arch"]
    E = ARCH[arch]["n_embd"]
    torch.manual_seed(seed)
    with torch.device(dev):
        if kind == "model_train":
            model = models.MVPFormerModel(_config(arch)).to(torch.bfloat16).train()
            head = models.MVPFormerHead(E, 2).to(torch.bfloat16)
            x = torch.randn(B, T, C, E, generator=gen).to(torch.bfloat16)
            labels = torch.randint(0, 2, (B,), generator=gen)
            buckets = [list(p for n, p in m.named_parameters() if not n.startswith("ln_2"))
                       for m in [*model.h, model.ln_f, model.positional_embedding, model.channel_embedding, head]]
            return dict(kind=kind, model=model, head=head, x=x, labels=labels, buckets=buckets)
        gen_task = kind == "next_state"
        cls = models.HMVPFormer if gen_task else models.ClassificationHMVPFormer
        task = cls(_config(arch), models.WaveEncoder(SEGMENT, E), models.MVPFormerHead(E, None if gen_task else 2),
                   num_negatives=NEGATIVES)
    task = task.to(torch.bfloat16).eval()
    if case["graph"]:
        task.mvpformer.enable_cuda_graph()
    state = dict(kind=kind, task=task, x=synthetic_ieeg(B, T, C, SEGMENT, seed=seed, device=dev))
    if gen_task:
        # any row of the batch but the target itself
        n = B * T * C
        neg = torch.randint(0, n - 1, (n, NEGATIVES), generator=gen, device=dev, dtype=torch.int32)
        neg += neg >= torch.arange(n, device=dev)[:, None]
        state["negatives"] = neg.view(B, T, C, NEGATIVES)
    return state


def run(state):
    kind = state["kind"]
    if kind == "attend":
        with torch.no_grad():
            return attentions.flashmvpa(*state["args"], True, state["scale"], window_size=WINDOW)
    if kind == "attend_train":
        o = attentions.flashmvpa(*state["args"], True, state["scale"], window_size=WINDOW)
        return (o.detach(),) + torch.autograd.grad(o, state["args"], state["d_o"])
    if kind == "classify":
        return state["task"].classify(state["x"])
    if kind == "next_state":
        return state["task"].next_state_logits(state["x"], negatives=state["negatives"])
    # training step: last hidden state -> classification readout -> loss -> gradients, one flat bucket per block
    out = state["model"](inputs_embeds=state["x"]).last_hidden_state
    logits = state["head"](out[:, -1].mean(dim=1))
    loss = torch.nn.functional.cross_entropy(logits.float(), state["labels"])
    grads = iter(torch.autograd.grad(loss, [p for b in state["buckets"] for p in b]))
    return [logits.detach()] + [torch.cat([next(grads).flatten() for _ in b]) for b in state["buckets"]]


# ---------------------------------------------------------------------------------------------------------------------
def _attention_flops(B, H, T, C, D, train):
    """Products over the pairs that the path needs: causal pairs for PV, windowed pairs for the content scores, and the two
    relative products; backward: dP and dV over causal pairs, S, dQ and dK over windowed pairs, three per relative product."""
    N = T * C
    causal = C * C * T * (T + 1) // 2
    windowed = C * C * (sum(min(t, WINDOW) + 1 for t in range(T - 1)) + T)
    fwd = 2 * D * (causal + windowed) + 2 * D * N * (T + C)
    bwd = 2 * D * (2 * causal + 3 * windowed) + 6 * D * N * (T + C)
    return B * H * (fwd + (bwd if train else 0))


def work(case):
    B, T, C = case["B"], case["T"], case["C"]
    if case["kind"] in ("attend", "attend_train"):
        H, Hkv, D = case["H"], case["Hkv"], case["D"]
        es = 2 if case["dtype"] == "bf16" else 4
        qo, kv, small = B * H * T * C * D, B * Hkv * T * C * D, Hkv * D * (3 + T + C)
        train = case["kind"] == "attend_train"
        # forward: q, k, v and the small tensors in, o out; a training pass also reads dO and writes dq, dk, dv and the rest
        values = 2 * qo + 2 * kv + small + (2 * qo + 2 * kv + small if train else 0)
        return {"bytes": es * values, "flops": _attention_flops(B, H, T, C, D, train)}
    a = ARCH[case["arch"]]
    E, I, L, H = a["n_embd"], a["n_inner"], a["n_layer"], a["n_head"]
    kv = E // H * a["n_head_kv"]
    tokens = B * T * C
    block = 2 * E * E + 2 * kv * E + 3 * I * E            # q, c_proj, k|v, gate, up, down
    rel = 2 * kv * E
    train = case["kind"] == "model_train"
    flops = (3 if train else 1) * L * (2 * tokens * block + 2 * (T + C) * kv * E) + L * _attention_flops(B, H, T, C, E // H, train)
    params = L * (block + rel + 3 * kv + E) + (T + C + 1) * E
    if train:
        return {"bytes": 2 * (2 * params + tokens * E), "flops": flops}
    coeffs = SEGMENT + 50                                  # wavelet coefficients of a segment
    flops += 2 * tokens * coeffs * E
    nbytes = 4 * tokens * SEGMENT + 2 * (params + coeffs * E)
    if case["kind"] == "next_state":
        flops += 2 * tokens * E * E + 6 * (B * (T - 1) * C) * NEGATIVES * E
        nbytes += 2 * E * E + 4 * tokens * NEGATIVES + 4 * B * (T - 1) * C * (NEGATIVES + 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Against the same path in 64 bits on the same inputs, the operator measures rel 2.5e-7 to 7e-7 in fp32 and 2.5e-3 to
    4.9e-3 (largest single difference 0.02 to 0.08 of the root mean square) in bf16; the bf16 models, whose every layer rounds
    to bf16, measure against fp32 arithmetic 0.1 to 1.2e-2 (class logits), 0.7 to 1.8e-2 (a training step: its two-class logits are
    the worst) and 2.1 to 2.3e-2 (next-state logits, differences of nearly orthogonal rows)."""
    if case.get("dtype") == "fp32":
        return {"rel": 3e-6, "max": 1e-4}
    if case["kind"] in ("attend", "attend_train"):
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 3e-2, "max": 0.6}
