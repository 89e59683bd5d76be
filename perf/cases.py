"""The single-GPU work of a program that uses this framework, as cases that can be timed and compared.

Five kinds of call, each through the package's public entry points:

``train``     ``LlamaTrainer.step`` on a batch in pinned host memory: forward, loss, backward, AdamW of every unit. Returns the
              loss, the fp32 master weights and the first moments (after the first step 0.1 x the gradient).
``tp_layer``  ``TensorParallelLayer.forward`` and ``.backward`` on a communicator of one rank: attention and MLP halves on the
              fused GEMM kernels, both norms, weight gradients.
``tp_mlp``    ``TensorParallelMLP.forward`` / ``TensorParallelMLPFp8.forward``: the MLP half in inference.
``moe``       ``MoELayer.forward`` (and ``.backward``): route, dispatch, grouped expert GEMMs, combine, in bf16 or with fp8
              gate/up weights.
``linear``    one projection as an inference loop calls it: ``train_ops.gemm`` in bf16, ``fp8.linear`` against a weight that was
              quantised once.

Sizes are those of the package's own model table (``LlamaConfig``), benchmark programs and tests; ``draw`` spreads them over
the ranges in between.
"""
from __future__ import annotations

import math
from dataclasses import replace

import torch

from rocm_systems_b200.comm import Communicator, get_unique_id
from rocm_systems_b200.models.llama import LlamaConfig, LlamaTrainer
from rocm_systems_b200.ops import fp8
from rocm_systems_b200.ops import train_ops as ops
from rocm_systems_b200.parallel.ep import MoELayer
from rocm_systems_b200.parallel.fsdp import AdamWConfig
from rocm_systems_b200.parallel.tp import TensorParallelLayer, TensorParallelMLP, TensorParallelMLPFp8


def listed():
    return [
        # The smallest training step there is (the configuration of the tests and of the smoke run): launches and host work.
        {"name": "train_tiny", "kind": "train", "model": "tiny", "layers": 2, "batch": 1, "seq": 128},
        # The benchmark's step, one sequence of 4096 tokens at the 8B model's full widths and vocabulary, with two of its layers
        # (with all of them the state does not fit the card three times).
        {"name": "train_8b_2_layers", "kind": "train", "model": "llama3-8b", "layers": 2, "batch": 1, "seq": 4096},
        # A smaller model (64-wide heads) on a batch whose rows are no multiple of anything.
        {"name": "train_1b_ragged", "kind": "train", "model": "llama3.2-1b", "layers": 4, "batch": 2, "seq": 999},
        # A whole tensor-parallel layer of the 8B model, forward and backward, one sequence.
        {"name": "tp_layer_8b", "kind": "tp_layer", "model": "llama3-8b", "rows": 4096, "seqs": 1},
        # The MLP half of that layer while decoding for 128 requests: the weights are read once, little arithmetic.
        {"name": "tp_mlp_decode", "kind": "tp_mlp", "dtype": "bf16", "rows": 128, "hidden": 4096, "ffn": 14336},
        # The MLP half of the tensor-parallel benchmark in fp8: 8192 rows, hidden 8192, a rank's 3584 columns.
        {"name": "tp_mlp_fp8_prefill", "kind": "tp_mlp", "dtype": "fp8", "rows": 8192, "hidden": 8192, "ffn": 3584},
        # A rank of the expert-parallel benchmark in prefill: 32 local experts, top-8, hidden 7168, 4096 tokens.
        {"name": "moe_prefill", "kind": "moe", "experts": 32, "hidden": 7168, "ffn": 2048, "topk": 8, "tokens": 4096, "fp8": False, "backward": False},
        # The same kind of layer while decoding for 64 requests, fp8 gate/up weights.
        {"name": "moe_decode_fp8", "kind": "moe", "experts": 32, "hidden": 4096, "ffn": 1024, "topk": 8, "tokens": 64, "fp8": True, "backward": False},
        # Training a mixture-of-experts layer: forward and backward with all weight gradients.
        {"name": "moe_train", "kind": "moe", "experts": 32, "hidden": 4096, "ffn": 1024, "topk": 8, "tokens": 4096, "fp8": False, "backward": True},
        # The 8B model's query/key/value projection while decoding for 16 requests.
        {"name": "linear_decode", "kind": "linear", "dtype": "bf16", "rows": 16, "n": 6144, "k": 4096},
        # Its gate/up projection in fp8 for a prompt of 4096 tokens, the activations quantised on the way.
        {"name": "fp8_linear_prefill", "kind": "linear", "dtype": "fp8", "rows": 4096, "n": 28672, "k": 4096},
        # Its down projection in fp8 while decoding for 32 requests.
        {"name": "fp8_linear_decode", "kind": "linear", "dtype": "fp8", "rows": 32, "n": 4096, "k": 14336},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_of(rng, lo, hi, unit):
    return max(lo, min(hi, (_log(rng, lo, hi) + unit // 2) // unit * unit))


def draw(rng):
    kind = rng.choice(["train", "tp_layer", "tp_mlp", "moe", "moe", "linear", "linear", "linear"])
    if kind == "train":
        model = rng.choice(["tiny", "llama3.2-1b", "llama3.2-3b", "llama3-8b"])
        batch = rng.randint(1, 3)
        seq = _log(rng, 32, {"tiny": 2048}.get(model, 3072) // batch)
        return {"kind": kind, "model": model, "layers": rng.randint(1, {"llama3-8b": 1, "llama3.2-3b": 2}.get(model, 4)), "batch": batch, "seq": seq}
    if kind == "tp_layer":
        model = rng.choice(["llama3.2-1b", "llama3.2-3b", "llama3-8b", "llama2-7b"])
        seqs = rng.randint(1, 2)
        return {"kind": kind, "model": model, "rows": _log_of(rng, 256, 4096, 256), "seqs": seqs}
    if kind == "tp_mlp":
        dtype = rng.choice(["bf16", "fp8"])
        return {"kind": kind, "dtype": dtype, "rows": _log_of(rng, 128, 8192, 128), "hidden": _log_of(rng, 1024, 8192, 128), "ffn": _log_of(rng, 1024, 4096, 128)}
    if kind == "moe":
        tokens = _log(rng, 1, 4096)
        fp8e = rng.random() < 0.4
        return {"kind": kind, "experts": 32, "hidden": 1024 * rng.randint(1, 4), "ffn": 128 * rng.randint(2, 12), "topk": rng.choice([2, 4, 8]), "tokens": tokens,
                "fp8": fp8e, "backward": not fp8e and rng.random() < 0.5}
    dtype = rng.choice(["bf16", "fp8"])
    unit = 128 if dtype == "fp8" else 8
    return {"kind": kind, "dtype": dtype, "rows": _log(rng, 1, 4096), "n": _log_of(rng, 512, 28672, 8), "k": _log_of(rng, 512, 14336, unit)}


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


_comm = None


def _communicator():
    """The program's one communicator (of one rank)."""
    global _comm
    if _comm is None:
        torch.cuda.set_device(0)
        _comm = Communicator(0, 1, get_unique_id(), 0)
    return _comm


class _Layer:
    """A parallel layer that gives its symmetric memory back when the program drops it."""

    def __init__(self, layer):
        self.layer = layer

    def __del__(self):
        self.layer.free()


def _model(case):
    cfg = LlamaConfig.by_name(case["model"])
    return replace(cfg, layers=case["layers"], seq_len=case["seq"]) if case["kind"] == "train" else cfg


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "train":
        cfg = _model(case)
        # the learning rate of the first steps of a warm-up, as the weights are random
        trainer = LlamaTrainer(cfg, None, torch.device("cuda", 0), opt=AdamWConfig(lr=1e-5), seed=seed)
        h = torch.Generator().manual_seed(seed)
        shape = (case["batch"], case["seq"])
        return {"kind": kind, "trainer": trainer, "tokens": torch.randint(0, cfg.vocab, shape, generator=h).pin_memory(),
                "targets": torch.randint(0, cfg.vocab, shape, generator=h).pin_memory()}
    if kind == "tp_layer":
        cfg = _model(case)
        layer = TensorParallelLayer(_communicator(), case["rows"], cfg.hidden, cfg.heads, cfg.kv_heads, cfg.ffn, case["rows"] // case["seqs"], seed=seed)
        return {"kind": kind, "held": _Layer(layer), "x": _randn(g, case["rows"], cfg.hidden), "dy": _randn(g, case["rows"], cfg.hidden, scale=1e-2)}
    if kind == "tp_mlp":
        cls = TensorParallelMLPFp8 if case["dtype"] == "fp8" else TensorParallelMLP
        layer = cls(_communicator(), case["rows"], case["hidden"], case["ffn"], seed=seed)
        return {"kind": kind, "held": _Layer(layer), "x": _randn(g, case["rows"], case["hidden"])}
    if kind == "moe":
        layer = MoELayer(_communicator(), case["experts"], case["hidden"], case["ffn"], case["topk"], case["tokens"], seed=seed, fp8_experts=case["fp8"])
        # some experts are more popular than others, as with a trained router
        logits = torch.randn(case["tokens"], case["experts"], device="cuda", generator=g) + 0.5 * torch.randn(case["experts"], device="cuda", generator=g)
        st = {"kind": kind, "held": _Layer(layer), "x": _randn(g, case["tokens"], case["hidden"]), "logits": logits}
        if case["backward"]:
            st["dy"] = _randn(g, case["tokens"], case["hidden"], scale=1e-2)
        return st
    x = _randn(g, case["rows"], case["k"])
    w = _randn(g, case["n"], case["k"], scale=0.02)
    if case["dtype"] == "fp8":
        wq, ws = fp8.quantize_weight(w)
        return {"kind": kind, "dtype": "fp8", "x": x, "wq": wq, "ws": ws}
    return {"kind": kind, "dtype": "bf16", "x": x, "w": w}


def run(state):
    kind = state["kind"]
    if kind == "train":
        t = state["trainer"]
        loss = t.step(state["tokens"], state["targets"])
        units = [t.embed, *t.layers, t.head]
        return {"loss": loss, "master": [u.master for u in units], "m": [u.m for u in units]}
    if kind == "tp_layer":
        layer = state["held"].layer
        y = layer.forward(state["x"])
        dx = layer.backward(state["dy"])
        return {"y": y, "dx": dx, "norms": dict(layer.grads), "attn": dict(layer.attn.grads), "mlp": dict(layer.mlp.grads)}
    if kind == "tp_mlp":
        return state["held"].layer.forward(state["x"])
    if kind == "moe":
        layer = state["held"].layer
        y = layer.forward(state["x"], state["logits"])
        if "dy" not in state:
            return y
        dx, dlogits = layer.backward(state["dy"])
        return {"y": y, "dx": dx, "dlogits": dlogits, "w": dict(layer.grads)}
    if state["dtype"] == "fp8":
        return fp8.linear(state["x"], state["wq"], state["ws"])
    return ops.gemm(state["x"], state["w"])


def work(case):
    kind = case["kind"]
    if kind == "train":
        cfg = _model(case)
        tokens = case["batch"] * case["seq"]
        # every parameter's master weight and two moments are read and written, its bf16 copy written
        return {"bytes": 26.0 * cfg.param_count() + 16.0 * tokens, "flops": cfg.flops_per_token() * tokens}
    if kind == "tp_layer":
        cfg = _model(case)
        rows, H, d = case["rows"], cfg.hidden, cfg.head_dim
        params = H * (cfg.heads + 2 * cfg.kv_heads) * d + H * H + 3 * H * cfg.ffn
        attn = 6 * (rows // case["seqs"]) * H * rows  # causal, forward and backward
        return {"bytes": 2.0 * (2 * params + 4 * rows * H), "flops": 6.0 * params * rows + attn}
    if kind == "tp_mlp":
        w = 3 * case["hidden"] * case["ffn"]
        return {"bytes": (1.0 if case["dtype"] == "fp8" else 2.0) * w + 4.0 * case["rows"] * case["hidden"], "flops": 2.0 * w * case["rows"]}
    if kind == "moe":
        E, H, f, k, T = case["experts"], case["hidden"], case["ffn"], case["topk"], case["tokens"]
        used = E * (1.0 - (1.0 - k / E) ** T)  # experts that see a token, with even routing
        per = used * f * H
        if case["backward"]:
            return {"bytes": 2.0 * 3 * per + 2.0 * 3 * E * f * H + 8.0 * T * H + 8.0 * T * E, "flops": 18.0 * T * k * f * H}
        return {"bytes": (2 + 2 if case["fp8"] else 6) * per + 4.0 * T * H + 4.0 * T * E, "flops": 6.0 * T * k * f * H}
    M, N, K = case["rows"], case["n"], case["k"]
    return {"bytes": 2.0 * M * K + (1.0 if case["dtype"] == "fp8" else 2.0) * N * K + 2.0 * M * N, "flops": 2.0 * M * N * K}


def tolerance(case):
    """About four times what another correct implementation at the same precision was measured to differ by."""
    kind = case["kind"]
    if kind == "train":
        # linear layers on cuBLAS instead, two steps: 6e-3 in the moments (single elements near zero by up to half the rms)
        return {"rel": 2e-2, "max": 0.95}
    if kind == "linear":
        # against float64 rounded once: 1.6e-4 (bf16 operands), 3e-5 (fp8 operands, whose products are exact in fp32); one bf16 step at most
        return {"rel": 7e-4 if case["dtype"] == "bf16" else 2e-4, "max": 0.04}
    if kind == "tp_mlp" and case["dtype"] == "fp8":
        # the same quantised arithmetic in PyTorch: 1e-4; an activation on a rounding boundary changes its fp8 code
        return {"rel": 1e-3, "max": 0.1}
    # the unfused compositions with intermediate results rounded to bf16 in other places: 4e-3 to 5e-3
    return {"rel": 1.6e-2, "max": 0.2}
