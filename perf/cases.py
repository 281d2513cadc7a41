"""Performance cases: what users of the framework run, with sizes, inputs, required work and tolerances.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare(case, seed)`` builds what
a user's program holds before the call, ``run(state)`` is one pass through the public entry points, ``work(case)`` the
bytes and operations a pass cannot do without and ``tolerance(case)`` how far two correct implementations may differ.

Kinds of cases:

* ``lm_step``: one optimisation step of a language model through ``TrainStep`` (forward, backward, AdamW; replayed from
  a captured graph as in a training loop).  Loss, gradients and master weights come out;
* ``lm_logits``: forward pass of a language model without gradients (scoring, prefill, evaluation);
* ``attention``: causal grouped-query attention, forward only or forward and backward;
* ``linear``: a linear layer in the input types next to bf16 (fp16, and fp32 under the fast-math policy), forward and
  backward;
* ``convnet``: a convolution / batch norm / pooling trunk in bf16, forward and backward.
"""
from __future__ import annotations

import math

import torch
from torch import nn

from incin_b200.core.policy import MathMode, policy_scope
from incin_b200.engine import TrainStep
from incin_b200.models.gpt2 import GPT2, GPT2Config
from incin_b200.models.llama import Llama, LlamaConfig
from incin_b200.nn import layers as L
from incin_b200.ops import functional as F
from incin_b200.ops.attention import flash_attention
from incin_b200.optim import AdamW, ParamStore

DEVICE = "cuda"


# ------------------------------------------------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # the training benchmark of the framework: GPT-2-small, micro-batch 8, full context
        {"name": "gpt2_small_step", "kind": "lm_step", "model": "gpt2-small", "layers": 12, "batch": 8, "seq": 1024},
        # fine-tuning on short ragged sequences: neither rows nor context are multiples of a tile
        {"name": "gpt2_small_step_ragged", "kind": "lm_step", "model": "gpt2-small", "layers": 12, "batch": 3, "seq": 517},
        # the smallest model of the repository: a step is many short launches
        {"name": "gpt2_tiny_step", "kind": "lm_step", "model": "gpt2-tiny", "layers": 2, "batch": 4, "seq": 128},
        # the two Llama widths of the repository on one GPU (fewer blocks than the full models, which are sharded)
        {"name": "llama_1b_step", "kind": "lm_step", "model": "llama-1b", "layers": 4, "batch": 4, "seq": 2048},
        {"name": "llama_3b_step", "kind": "lm_step", "model": "llama-3b", "layers": 2, "batch": 1, "seq": 4096},
        # scoring one short prompt: latency of a forward pass
        {"name": "gpt2_small_logits_short", "kind": "lm_logits", "model": "gpt2-small", "layers": 12, "batch": 1, "seq": 61},
        # evaluation over a batch of full documents
        {"name": "gpt2_small_logits_batch", "kind": "lm_logits", "model": "gpt2-small", "layers": 12, "batch": 8, "seq": 1000},
        # the attention benchmark of the framework, forward and backward
        {"name": "attention_train", "kind": "attention", "batch": 8, "seq": 4096, "heads": 32, "kv_heads": 32,
         "head_dim": 128, "backward": True},
        # prefill of one long odd-sized document with the grouped heads of the 3B model
        {"name": "attention_prefill", "kind": "attention", "batch": 1, "seq": 8191, "heads": 24, "kv_heads": 8,
         "head_dim": 128, "backward": False},
        # mixed precision in fp16
        {"name": "linear_fp16", "kind": "linear", "dtype": "fp16", "rows": 4096, "n_in": 768, "n_out": 3072},
        # fp32 models with the fast-math policy
        {"name": "linear_fp32_fast", "kind": "linear", "dtype": "fp32", "rows": 8184, "n_in": 1024, "n_out": 1000},
        # image trunk
        {"name": "convnet", "kind": "convnet", "batch": 64, "channels": 64, "height": 32, "width": 32},
    ]


def _log_int(rng, lo: int, hi: int, step: int = 1) -> int:
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(max(int(round(v / step)) * step, lo), hi)


def draw(rng) -> dict:
    kind = rng.choice(["lm_step", "lm_step", "lm_logits", "attention", "attention", "linear", "convnet"])
    if kind == "lm_step":
        model = rng.choice(["gpt2-small", "gpt2-tiny", "llama-1b", "llama-3b"])
        if model == "gpt2-tiny":
            return {"kind": kind, "model": model, "layers": 2, "batch": rng.randint(1, 8), "seq": _log_int(rng, 17, 128)}
        if model == "gpt2-small":
            return {"kind": kind, "model": model, "layers": rng.randint(2, 12), "batch": rng.randint(1, 8),
                    "seq": _log_int(rng, 100, 1024)}
        # tokens x layers stays below the listed cases'
        tokens, layers = (8192, rng.randint(1, 4)) if model == "llama-1b" else (4096, rng.randint(1, 2))
        seq = _log_int(rng, 256, 2048 if model == "llama-1b" else 4096)
        return {"kind": kind, "model": model, "layers": layers, "batch": rng.randint(1, max(1, tokens // seq)), "seq": seq}
    if kind == "lm_logits":
        return {"kind": kind, "model": "gpt2-small", "layers": 12, "batch": _log_int(rng, 1, 8), "seq": _log_int(rng, 16, 1000)}
    if kind == "attention":
        # the head configurations of the repository: attention benchmark, GPT-2-small, Llama 1.1B, Llama 3B
        heads, kv_heads, head_dim = rng.choice([(32, 32, 128), (12, 12, 64), (32, 4, 64), (24, 8, 128)])
        seq = _log_int(rng, 128, 8191)
        # no more than the listed benchmark: batch x heads x seq^2
        batch = max(1, min(rng.randint(1, 8), int(8 * 32 * 4096 ** 2 / (heads * seq ** 2))))
        return {"kind": kind, "batch": batch, "seq": seq, "heads": heads, "kv_heads": kv_heads,
                "head_dim": head_dim, "backward": rng.random() < 0.5}
    if kind == "linear":
        dtype = rng.choice(["fp16", "fp32"])
        return {"kind": kind, "dtype": dtype, "rows": _log_int(rng, 64, 8192), "n_in": _log_int(rng, 256, 4096, 8),
                "n_out": _log_int(rng, 64, 4096, 8)}
    return {"kind": kind, "batch": _log_int(rng, 4, 64), "channels": rng.choice([16, 32, 64]),
            "height": rng.randint(14, 40), "width": rng.randint(14, 40)}


# ----------------------------------------------------------------------------------------------------------- prepare
def _config(case: dict):
    cfg = {"gpt2-small": GPT2Config.small, "gpt2-tiny": GPT2Config.tiny, "llama-1b": LlamaConfig.llama_1b,
           "llama-3b": LlamaConfig.llama_3b}[case["model"]]()
    cfg.n_layer = case["layers"]
    return cfg


def _model(case: dict, cfg, gen: torch.Generator) -> nn.Module:
    """The model on the GPU with weights ~ N(0, init_std), biases 0 and gains 1, drawn on the device."""
    base = GPT2 if isinstance(cfg, GPT2Config) else Llama

    class Seeded(base):
        def reset_parameters(self, seed: int = 0) -> None:
            with torch.no_grad():
                for p in self.parameters():
                    if p.dim() >= 2:
                        p.normal_(0.0, cfg.init_std, generator=gen)

    with torch.device(DEVICE):
        return Seeded(cfg)


def _tokens(case: dict, cfg, gen: torch.Generator) -> torch.Tensor:
    return torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=gen, device=DEVICE)


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]

    def randn(*shape, dtype=torch.bfloat16, scale=1.0):
        return (torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float32) * scale).to(dtype)

    if kind == "lm_step":
        cfg = _config(case)
        model = _model(case, cfg, gen)
        store = ParamStore(model.named_parameters())
        opt = AdamW(store, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1)
        step = TrainStep(model, opt)
        tok, tgt = _tokens(case, cfg, gen), _tokens(case, cfg, gen)
        # a training loop in progress: the step has been captured (two eager calls, then the capture), and the weights
        # and moments are put back to where they were before these calls
        master = store.master.clone()
        for _ in range(3):
            step(tok, tgt)
        store.master.copy_(master)
        store.sync_shadow_from_master()
        opt.m.zero_()
        opt.v.zero_()
        opt.step_count = 0
        return {"case": case, "step": step, "store": store, "tok": tok, "tgt": tgt}
    if kind == "lm_logits":
        cfg = _config(case)
        model = _model(case, cfg, gen).to(torch.bfloat16)
        return {"case": case, "model": model, "tok": _tokens(case, cfg, gen)}
    if kind == "attention":
        B, T, D = case["batch"], case["seq"], case["head_dim"]
        q, k, v = (randn(B, T, h, D) for h in (case["heads"], case["kv_heads"], case["kv_heads"]))
        state = {"case": case, "q": q, "k": k, "v": v}
        if case["backward"]:
            for t in (q, k, v):
                t.requires_grad_()
            state["dout"] = randn(B, T, case["heads"], D)
        return state
    if kind == "linear":
        dtype = {"fp16": torch.float16, "fp32": torch.float32}[case["dtype"]]
        x = randn(case["rows"], case["n_in"], dtype=dtype).requires_grad_()
        layer = L.Linear(case["n_in"], case["n_out"]).to(DEVICE, dtype)
        with torch.no_grad():
            layer.weight.copy_(randn(case["n_out"], case["n_in"], scale=case["n_in"] ** -0.5, dtype=dtype))
            layer.bias.copy_(randn(case["n_out"], scale=case["n_in"] ** -0.5, dtype=dtype))
        return {"case": case, "x": x, "layer": layer, "dout": randn(case["rows"], case["n_out"], dtype=dtype)}
    C = case["channels"]
    # (no convolution bias: the batch norm behind it would take it out again)
    net = L.seq(L.Conv2d(C, C, 3, padding=1, bias=False), L.BatchNorm2d(C), L.ReLU(), L.MaxPool2d(2),
                L.Conv2d(C, 2 * C, 3, padding=1, bias=False), L.BatchNorm2d(2 * C), L.ReLU(),
                L.AdaptiveAvgPool2d(4)).to(DEVICE)
    for m in net:
        if isinstance(m, L.Conv2d):
            m.to(torch.bfloat16)
            with torch.no_grad():
                m.weight.copy_(randn(*m.weight.shape, scale=(9 * C) ** -0.5))
    x = randn(case["batch"], C, case["height"], case["width"]).requires_grad_()
    return {"case": case, "net": net, "x": x, "dout": randn(case["batch"], 2 * C, 4, 4)}


# --------------------------------------------------------------------------------------------------------------- run
def run(state: dict):
    kind = state["case"]["kind"]
    if kind == "lm_step":
        loss = state["step"](state["tok"], state["tgt"])
        return {"loss": loss, "grad": state["store"].grad, "weights": state["store"].master}
    if kind == "lm_logits":
        with torch.no_grad():
            return state["model"](state["tok"])
    if kind == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        if not state["case"]["backward"]:
            with torch.no_grad():
                return flash_attention(q, k, v)
        out = flash_attention(q, k, v)
        return (out.detach(), *torch.autograd.grad(out, (q, k, v), state["dout"]))
    if kind == "linear":
        layer, x = state["layer"], state["x"]
        fast = MathMode.FAST if state["case"]["dtype"] == "fp32" else MathMode.PRECISE
        with policy_scope(math=fast):
            y = F.linear(x, layer.weight, layer.bias)
            grads = torch.autograd.grad(y, (x, layer.weight, layer.bias), state["dout"])
        return (y.detach(), *grads)
    net, x = state["net"], state["x"]
    y = net(x)
    return (y.detach(), *torch.autograd.grad(y, (x, *net.parameters()), state["dout"]))


# -------------------------------------------------------------------------------------------------------------- work
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("lm_step", "lm_logits"):
        cfg = _config(case)
        n, rows = cfg.num_params(), case["batch"] * case["seq"]
        forward = cfg.flops_per_token(case["seq"]) / 3.0 * rows      # matmuls and the causal half of attention
        if kind == "lm_logits":
            return {"bytes": 2 * n + 8 * rows + 2 * rows * cfg.vocab_size, "flops": forward}
        # AdamW: master weights and two moments read and written, the gradient written, the bf16 weights read and
        # written; plus the tokens
        return {"bytes": n * (6 * 4 + 4 + 2 * 2) + 16 * rows, "flops": 3.0 * forward}
    if kind == "attention":
        B, T, H, Hk, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        pair = 2.0 * B * H * D * T * (T + 1) / 2        # one product over the causal half
        io = 2 * B * T * D * (2 * H + 2 * Hk)           # q, k, v in, out written
        if not case["backward"]:
            return {"bytes": io, "flops": 2 * pair}
        return {"bytes": io + 2 * B * T * D * (2 * H + 2 * Hk), "flops": 7 * pair}
    if kind == "linear":
        R, I, O = case["rows"], case["n_in"], case["n_out"]
        size = 2 if case["dtype"] == "fp16" else 4
        # x, w, b, dout in; y, dx, dw, db out
        return {"bytes": size * (2 * R * I + 2 * I * O + 2 * R * O + 2 * O), "flops": 6.0 * R * I * O}
    N, C, H, W = case["batch"], case["channels"], case["height"], case["width"]
    first, second = N * H * W * C * 9 * C, N * (H // 2) * (W // 2) * C * 9 * 2 * C
    return {"bytes": 2 * (2 * N * C * H * W + 2 * N * 2 * C * 16 + 2 * (9 * C * C + 18 * C * C)),
            "flops": 6.0 * (first + second)}


# --------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case: dict) -> dict:
    """Each about four times what was measured on a B200 (relative 2-norm): a bf16 training step against the same model
    in fp32 0.005-0.016 (two runs of the step among themselves 0.004: fp32 atomics), bf16 logits 0.009, bf16 attention
    and its gradients against 64 bits 0.0025, fp16 linear 0.0002, fp32 multiplied as tf32 0.0008.  The trunk's input
    gradient is 0.07 from 64 bits, because a rounded activation moves some gradients to another element of their pooling
    window or past the ReLU."""
    return {"lm_step": {"rel": 3e-2}, "lm_logits": {"rel": 3e-2}, "attention": {"rel": 1e-2},
            "linear": {"rel": 1e-3 if case.get("dtype") == "fp16" else 3e-3},
            "convnet": {"rel": 5e-2, "max": 0.9}}[case["kind"]]
