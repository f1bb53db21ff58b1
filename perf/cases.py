"""Performance cases of the framework on one GPU, through its public entry points.

Every case is a dict of plain values; ``kind`` names the entry point:

  a2a        ``MoEAllToAll.dispatch_scale_combine``: the MoE round trip with a scale as the expert
  gemm_rs    ``GemmRS.__call__``: GEMM + reduce-scatter
  ag_gemm    ``AGGemm.__call__``: all-gather + GEMM
  rs_host    ``GemmRS.run_from_host``: the same op with its activations and its result in pinned host memory
  mlp        ``SequenceParallelMLP``: forward pass
  mlp_train  ``TrainableSequenceParallelMLP``: forward and backward pass
  moe        ``MoELayer``: forward pass over real expert MLPs
  moe_train  ``TrainableMoELayer``: forward and backward pass

``prepare`` makes what a program holds before a step (inputs, weights, the op's context), ``run`` does one
step, ``work`` counts what the step cannot do without, ``tolerance`` says how close two correct
implementations of the same precision come.
"""
from __future__ import annotations

import math

import torch

from kernel_b200.models import MoELayer, SequenceParallelMLP, TrainableMoELayer, TrainableSequenceParallelMLP
from kernel_b200.ops.dispatch_combine import MoEAllToAll
from kernel_b200.ops.gemm import AGGemm, GemmRS

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEMENT_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
SCALE = {"identity": 0, "rank": 1, "expert": 2}


def listed():
    return [
        # MoE round trip: one token of a decoding step (the smallest call: launch and latency only)
        {"name": "a2a_decode_1", "kind": "a2a", "experts": 256, "topk": 8, "hidden": 7168, "capacity": 1, "tokens": 1,
         "dtype": "bf16", "scale": "expert"},
        # ... a ragged batch below the context's capacity, fp16, hidden size off the powers of two
        {"name": "a2a_ragged_fp16", "kind": "a2a", "experts": 128, "topk": 4, "hidden": 2880, "capacity": 128, "tokens": 101,
         "dtype": "fp16", "scale": "rank"},
        # ... a prefill batch, the benchmark's size on one GPU
        {"name": "a2a_prefill_2048", "kind": "a2a", "experts": 256, "topk": 8, "hidden": 7168, "capacity": 2048, "tokens": 2048,
         "dtype": "bf16", "scale": "expert"},
        # output projection of a decoding step: few rows, the weight matrix is the traffic
        {"name": "gemm_rs_decode_64", "kind": "gemm_rs", "m": 64, "n": 7168, "k": 18432, "bias": False},
        # a mid-size projection whose N and K are not multiples of the tile
        {"name": "gemm_rs_mid", "kind": "gemm_rs", "m": 2048, "n": 2880, "k": 2880, "bias": True},
        # the benchmark's GEMM + reduce-scatter
        {"name": "gemm_rs_flagship", "kind": "gemm_rs", "m": 8192, "n": 8192, "k": 29568, "bias": True},
        # input projection of a prefill batch
        {"name": "ag_gemm_prefill", "kind": "ag_gemm", "m": 4096, "n": 14336, "k": 4096, "bias": True},
        # activations that arrive from and return to the host
        {"name": "rs_host_stream", "kind": "rs_host", "m": 2048, "n": 4096, "k": 7168, "bias": True},
        # dense MLP, inference on a small batch
        {"name": "mlp_forward_256", "kind": "mlp", "tokens": 256, "hidden": 4096, "ffn": 14336, "act": "gelu"},
        # dense MLP, training step of the step benchmark's default size (the largest case)
        {"name": "mlp_train_flagship", "kind": "mlp_train", "tokens": 8192, "hidden": 8192, "ffn": 29568, "act": "gelu"},
        # MoE layer, inference on a small batch: most experts see a few rows
        {"name": "moe_forward_32", "kind": "moe", "experts": 64, "topk": 6, "hidden": 2048, "ffn": 1024, "tokens": 32},
        # MoE layer, training step
        {"name": "moe_train_1024", "kind": "moe_train", "experts": 64, "topk": 8, "hidden": 2048, "ffn": 1024, "tokens": 1024},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], uniform over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step, max(-(-lo // step), round(v / step))) * step


# Inclusive bounds of the sizes a case of each kind is drawn from.
MAX_GEMM_FLOPS = 2 * 8192 * 8192 * 29568
MAX_HOST_BYTES = 256 << 20      # activations in plus result out of one rs_host call
MAX_EXPERT_WEIGHTS = 1 << 28    # experts * hidden * ffn, one of the two matrices


def draw(rng):
    kind = rng.choice(["a2a", "a2a", "gemm_rs", "gemm_rs", "ag_gemm", "rs_host", "mlp", "mlp_train", "moe", "moe_train"])
    if kind == "a2a":
        experts = rng.choice([8, 32, 64, 128, 256])
        topk = rng.choice([k for k in (1, 2, 4, 6, 8) if k <= experts])
        tokens = _log(rng, 1, 2048)
        return {"kind": kind, "experts": experts, "topk": topk, "hidden": _log(rng, 1024, 7168, 8),
                "capacity": rng.choice([tokens, min(2048, tokens + tokens // 3 + 1)]), "tokens": tokens,
                "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"]), "scale": rng.choice(["expert", "rank", "identity"])}
    if kind in ("gemm_rs", "ag_gemm"):
        while True:
            m, n, k = _log(rng, 16, 16384), _log(rng, 1024, 29568, 8), _log(rng, 1024, 29568, 8)
            if 2 * m * n * k <= MAX_GEMM_FLOPS:
                return {"kind": kind, "m": m, "n": n, "k": k, "bias": rng.random() < 0.5}
    if kind == "rs_host":
        while True:
            m, n, k = _log(rng, 256, 8192, 4), _log(rng, 1024, 8192, 8), _log(rng, 1024, 8192, 8)
            if 2 * m * (n + k) <= MAX_HOST_BYTES:
                return {"kind": kind, "m": m, "n": n, "k": k, "bias": rng.random() < 0.5}
    if kind in ("mlp", "mlp_train"):
        train = kind == "mlp_train"
        while True:
            tokens = _log(rng, 128, 8192, 8) if train else _log(rng, 1, 8192)
            hidden, ffn = _log(rng, 1024, 8192, 8), _log(rng, 2048, 29568, 8)
            if 2 * tokens * hidden * ffn <= MAX_GEMM_FLOPS // (4 if train else 1):
                return {"kind": kind, "tokens": tokens, "hidden": hidden, "ffn": ffn, "act": rng.choice(["gelu", "silu", "relu"])}
    while True:
        experts = rng.choice([8, 16, 32, 64, 128])
        hidden, ffn = _log(rng, 512, 4096, 8), _log(rng, 512, 4096, 8)
        if experts * hidden * ffn <= MAX_EXPERT_WEIGHTS:
            tokens = _log(rng, 64, 4096) if kind == "moe_train" else _log(rng, 1, 4096)
            return {"kind": kind, "experts": experts, "topk": rng.choice([1, 2, 4, 6, 8]), "hidden": hidden, "ffn": ffn,
                    "tokens": tokens}


class _Random:
    """Seeded normal tensors on the GPU."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.device).manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        out = torch.empty(shape, dtype=dtype, device=self.device)
        return out.normal_(0.0, std, generator=self.g)

    def routing(self, tokens, experts, topk):
        """Distinct expert ids drawn uniformly per token and softmax weights over normal logits."""
        scores = torch.rand((tokens, experts), device=self.device, generator=self.g)
        indices = scores.argsort(dim=1)[:, :topk].to(torch.int32).contiguous()
        return indices, torch.softmax(self.normal(tokens, topk, dtype=torch.float32), dim=-1)


def prepare(case, seed):
    r, kind = _Random(seed), case["kind"]
    s = {"kind": kind}
    if kind == "a2a":
        s["ctx"] = MoEAllToAll(case["experts"], case["topk"], case["hidden"], case["capacity"], dtype=DTYPES[case["dtype"]],
                               device=r.device)
        s["x"] = r.normal(case["tokens"], case["hidden"], dtype=DTYPES[case["dtype"]])
        s["indices"], s["weights"] = r.routing(case["tokens"], case["experts"], case["topk"])
        s["scale"] = SCALE[case["scale"]]
    elif kind in ("gemm_rs", "ag_gemm", "rs_host"):
        m, n, k = case["m"], case["n"], case["k"]
        s["ctx"] = AGGemm(m, k, device=r.device) if kind == "ag_gemm" else GemmRS(m, n, device=r.device)
        a = r.normal(m, k)
        s["w"] = r.normal(n, k, std=k ** -0.5)
        s["bias"] = r.normal(n, std=0.02) if case["bias"] else None
        if kind == "rs_host":
            s["a"] = a.cpu().pin_memory()
            s["out"] = torch.empty((m, n), dtype=torch.bfloat16).pin_memory()
        else:
            s["a"] = a
    elif kind in ("mlp", "mlp_train"):
        tokens, hidden, ffn = case["tokens"], case["hidden"], case["ffn"]
        w1, w2 = r.normal(ffn, hidden, std=hidden ** -0.5), r.normal(hidden, ffn, std=ffn ** -0.5)
        b1, b2 = r.normal(ffn, std=0.02), r.normal(hidden, std=0.02)
        s["x"] = r.normal(tokens, hidden)
        if kind == "mlp":
            s["layer"] = SequenceParallelMLP(tokens, hidden, w1, w2, b1, b2, activation=case["act"])
        else:
            s["layer"] = layer = TrainableSequenceParallelMLP(tokens, hidden, ffn, activation=case["act"], device=r.device)
            with torch.no_grad():
                for p, v in ((layer.up.weight, w1), (layer.up.bias, b1), (layer.down.weight, w2), (layer.down.bias, b2)):
                    p.copy_(v)
            s["x"].requires_grad_(True)
            s["dy"] = r.normal(tokens, hidden)
    else:
        experts, topk, hidden, ffn, tokens = (case[key] for key in ("experts", "topk", "hidden", "ffn", "tokens"))
        w_up, w_down = r.normal(experts, ffn, hidden, std=hidden ** -0.5), r.normal(experts, hidden, ffn, std=ffn ** -0.5)
        s["x"] = r.normal(tokens, hidden)
        s["indices"], s["weights"] = r.routing(tokens, experts, topk)
        if kind == "moe":
            s["layer"] = MoELayer(experts, topk, hidden, tokens, w_up, w_down)
        else:
            s["layer"] = layer = TrainableMoELayer(experts, topk, hidden, ffn, tokens, device=r.device)
            with torch.no_grad():
                layer.w_up.copy_(w_up)
                layer.w_down.copy_(w_down)
            s["x"].requires_grad_(True)
            s["weights"].requires_grad_(True)
            s["dy"] = r.normal(tokens, hidden)
    return s


def _training_step(layer, leaves, dy, *inputs):
    """Forward and backward from cleared gradients; the output and the gradient of every leaf."""
    for p in leaves:
        p.grad = None
    y = layer(*inputs)
    y.backward(dy)
    return [y.detach()] + [p.grad for p in leaves]


def run(s):
    kind = s["kind"]
    if kind == "a2a":
        return s["ctx"].dispatch_scale_combine(s["x"], s["indices"], s["weights"], s["scale"])
    if kind in ("gemm_rs", "ag_gemm"):
        return s["ctx"](s["a"], s["w"], s["bias"])
    if kind == "rs_host":
        return s["ctx"].run_from_host(s["a"], s["w"], s["bias"], out_host=s["out"])
    if kind == "mlp":
        return s["layer"](s["x"])
    if kind == "mlp_train":
        return _training_step(s["layer"], [s["x"], *s["layer"].parameters()], s["dy"], s["x"])
    if kind == "moe":
        return s["layer"](s["x"], s["indices"], s["weights"])
    return _training_step(s["layer"], [s["x"], s["weights"], *s["layer"].parameters()], s["dy"], s["x"], s["indices"], s["weights"])


def work(case):
    """Every input read once and every output written once; the products' multiplications and additions."""
    kind = case["kind"]
    if kind == "a2a":
        t, k, h = case["tokens"], case["topk"], case["hidden"]
        return {"bytes": 2 * t * h * ELEMENT_BYTES[case["dtype"]] + 8 * t * k, "flops": 2 * t * k * h}
    if kind in ("gemm_rs", "ag_gemm", "rs_host"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n + (n if case["bias"] else 0)), "flops": 2 * m * n * k}
    if kind in ("mlp", "mlp_train"):
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        if kind == "mlp":
            return {"bytes": 2 * (2 * t * h + 2 * h * f + h + f), "flops": 4 * t * h * f}
        return {"bytes": 2 * (4 * t * h + 4 * h * f + 2 * (h + f)), "flops": 12 * t * h * f}
    e, k, h, f, t = (case[key] for key in ("experts", "topk", "hidden", "ffn", "tokens"))
    touched = e * (1.0 - (1.0 - k / e) ** t)  # expected number of experts that receive a row
    if kind == "moe":
        return {"bytes": 2 * (2 * t * h + 2 * touched * h * f) + 8 * t * k, "flops": 4 * t * k * h * f}
    return {"bytes": 2 * (4 * t * h + 2 * touched * h * f + 2 * e * h * f) + 12 * t * k, "flops": 12 * t * k * h * f}


def tolerance(case):
    if case["kind"] == "a2a":
        return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}
    # products: bf16 operands, fp32 accumulation, one bf16 rounding per result; the layers round between their products too
    return {"rel": 1e-2}
