"""The work this backend is measured on: what programs ask of it through its public entry points.

Five families, each over a range of sizes:

  chain, norm, mlp    functions of a user's own behind `lumen_b200.compile`: a loop-fused element-wise / row-sum chain, a
                      residual layer norm and an MLP block, the latter two with their backward by `lumen_b200.autograd`
  matmul              the three products of `F.matmul` and its backward through `lumen_b200.runtime.gemm`
  attention           `lumen_b200.runtime.attention_forward` / `attention_backward`: training at both head dims of the
                      tensor-core kernels, prefill with grouped heads, decode of one token against a cache
  step                `lumen_b200.transformer.TrainStep`: forward, backward and optimizer update of a decoder transformer

Inputs are made on the GPU from the seed alone. A compiled function is kept per signature, as a program keeps it that
compiles once and calls often; a training step keeps its own plan.
"""

import functools
import math

import numpy as np
import torch

import lumen_b200
from lumen_b200 import autograd, prims, runtime, transformer
from lumen_b200 import functional as F
from lumen_b200.runtime import TORCH_DTYPES

ITEM = {"float32": 4, "bfloat16": 2, "float16": 2}


def listed():
    return [
        # A handful of rows: one step of a small model or of a server with one request. Bound by what a call costs.
        {"name": "chain_small_f32", "kind": "chain", "rows": 64, "cols": 256, "dtype": "float32"},
        # The benchmark's own chain, larger than the L2: memory bandwidth.
        {"name": "chain_f32", "kind": "chain", "rows": 16384, "cols": 4096, "dtype": "float32"},
        # The same in bfloat16 on a width that is no multiple of a 16-byte line (an unpadded vocabulary or feature count).
        {"name": "chain_odd_bf16", "kind": "chain", "rows": 5000, "cols": 3001, "dtype": "bfloat16"},
        # Residual add + layer norm, forward and backward, of 8192 tokens: row reductions both ways and the column sums
        # of the weight gradients.
        {"name": "norm_train_bf16", "kind": "norm", "rows": 8192, "cols": 1024, "dtype": "bfloat16"},
        # One MLP block forward and backward on one short ragged sequence (fine-tuning at batch 1): six small products.
        {"name": "mlp_train_small_bf16", "kind": "mlp", "tokens": 200, "width": 1024, "hidden": 4096, "dtype": "bfloat16"},
        # The benchmark's matmul and its backward.
        {"name": "matmul_train_8192", "kind": "matmul", "m": 8192, "n": 8192, "k": 8192, "dtype": "bfloat16"},
        # Attention of the 12-layer model (16 heads x 64, sequence 2048), forward and backward, a rank's eight sequences,
        # in the mode the benchmark trains in.
        {"name": "attention_train_d64", "kind": "attention", "batch": 8, "heads": 16, "kv_heads": 16, "queries": 2048, "keys": 2048,
         "dim": 64, "causal": True, "backward": True, "deterministic": False},
        # The benchmark's attention at head dim 128.
        {"name": "attention_train_d128", "kind": "attention", "batch": 8, "heads": 32, "kv_heads": 32, "queries": 4096, "keys": 4096,
         "dim": 128, "causal": True, "backward": True, "deterministic": True},
        # Prefill of two prompts of a length nobody rounded, four query heads to a key head.
        {"name": "attention_prefill_gqa", "kind": "attention", "batch": 2, "heads": 32, "kv_heads": 8, "queries": 1531, "keys": 1531,
         "dim": 128, "causal": True, "backward": False, "deterministic": True},
        # Decode: one new token of sixteen sequences against a cache of 4097 keys. The cache is read once: bandwidth.
        {"name": "attention_decode_gqa", "kind": "attention", "batch": 16, "heads": 32, "kv_heads": 8, "queries": 1, "keys": 4097,
         "dim": 128, "causal": True, "backward": False, "deterministic": True},
        # The 2-layer float32 training step the parity tests hold: small kernels, launches and exact CUDA-core products.
        {"name": "step_2layer_f32", "kind": "step", "layers": 2, "width": 128, "heads": 4, "hidden": 512, "vocab": 256, "seq": 64,
         "batch": 8, "dtype": "float32", "optimizer": "sgd", "deterministic": True},
        # The benchmark model's training step at its full width, half its depth and one of eight ranks' share of the batch.
        {"name": "step_6layer_bf16", "kind": "step", "layers": 6, "width": 1024, "heads": 16, "hidden": 4096, "vocab": 32768,
         "seq": 2048, "batch": 8, "dtype": "bfloat16", "optimizer": "sgd", "deterministic": False},
    ]


def _size(rng, low, high, multiple=1):
    """A size spread over the logarithm of [low, high], a multiple of `multiple`."""
    n = int(math.exp(rng.uniform(math.log(low), math.log(high))))
    return max(low, n // multiple * multiple)


def draw(rng):
    kind = rng.choice(["chain", "norm", "mlp", "matmul", "train", "train", "prefill", "decode", "step_f32", "step_bf16"])
    if kind == "chain":
        cols = _size(rng, 64, 16384, rng.choice([1, 8, 64]))
        return {"kind": "chain", "rows": max(1, _size(rng, 1 << 14, 1 << 26) // cols), "cols": cols, "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "norm":
        cols = _size(rng, 128, 8192, rng.choice([1, 8, 64]))
        return {"kind": "norm", "rows": max(1, _size(rng, 1 << 14, 1 << 25) // cols), "cols": cols, "dtype": rng.choice(["float32", "bfloat16"])}
    if kind == "mlp":
        width = _size(rng, 128, 2048, 8)
        return {"kind": "mlp", "tokens": _size(rng, 16, 8192), "width": width, "hidden": 4 * width, "dtype": rng.choice(["bfloat16", "float16"])}
    if kind == "matmul":
        return {"kind": "matmul", "m": _size(rng, 64, 8192), "n": _size(rng, 64, 8192, 8), "k": _size(rng, 64, 8192, 8),
                "dtype": rng.choice(["bfloat16", "float16"])}
    if kind in ("train", "prefill"):
        dim, seq = rng.choice([64, 128]), _size(rng, 64, 4096)
        heads = rng.choice([4, 8, 16, 32])
        most = max(1, min(32, int(8 * 32 * 4096 * 4096 * 128 / (heads * seq * seq * dim)) // 2))
        return {"kind": "attention", "batch": _size(rng, 1, most), "heads": heads, "kv_heads": heads // rng.choice([1, 1, 2, 4]),
                "queries": seq, "keys": seq, "dim": dim, "causal": rng.random() < 0.75, "backward": kind == "train",
                "deterministic": rng.random() < 0.5}
    if kind == "decode":
        kv = rng.choice([1, 2, 4, 8, 16])
        return {"kind": "attention", "batch": _size(rng, 1, 32), "heads": kv * rng.choice([1, 2, 4, 8]), "kv_heads": kv,
                "queries": rng.choice([1, 1, 1, 2, 4]), "keys": _size(rng, 128, 16384), "dim": rng.choice([64, 128]), "causal": True,
                "backward": False, "deterministic": True}
    if kind == "step_f32":
        heads = rng.choice([2, 4])
        return {"kind": "step", "layers": rng.choice([1, 2]), "width": 32 * heads, "heads": heads, "hidden": 128 * heads,
                "vocab": _size(rng, 64, 512, 4), "seq": _size(rng, 16, 128, 4), "batch": _size(rng, 1, 8), "dtype": "float32",
                "optimizer": rng.choice(["sgd", "adamw"]), "deterministic": rng.random() < 0.5}
    heads = rng.choice([4, 8, 12, 16])
    return {"kind": "step", "layers": rng.choice([1, 2, 3, 4]), "width": 64 * heads, "heads": heads, "hidden": 256 * heads,
            "vocab": _size(rng, 1024, 32768, 8), "seq": _size(rng, 128, 2048, 8), "batch": _size(rng, 1, 8), "dtype": "bfloat16",
            "optimizer": "sgd", "deterministic": rng.random() < 0.5}


# ---- the programs a user writes -----------------------------------------------------------------------------------
def chain(x, g, b):
    y = F.relu(x * g + b)
    return y, prims.reduce_sum(y * y, (1,), "float32")


def norm_train(x, r, w, b, dy):
    """Residual add and layer norm with float32 statistics, and the gradients of the sum, the scale and the bias."""

    def forward(a, res, scale, bias):
        s = a + res
        return F.layer_norm(s.to("float32"), scale.to("float32"), bias.to("float32")).to(a.dtype)

    y, pull = autograd.vjp(forward, x, r, w, b)
    dx, _, dw, db = pull(dy)  # both operands of the sum have the same gradient
    return y, dx, dw, db


def mlp_train(x, w1, w2, dy):
    """`x + relu(x w1) w2` and its gradients; products accumulate in float32 and are rounded once."""

    def forward(a, u, v):
        h = F.relu(F.matmul(a, u, "float32", a.dtype))
        return a + F.matmul(h, v, "float32", a.dtype)

    y, pull = autograd.vjp(forward, x, w1, w2)
    return (y, *pull(dy))


@functools.lru_cache(maxsize=None)
def compiled(program):
    return lumen_b200.compile(program)


PROGRAMS = {"chain": chain, "norm": norm_train, "mlp": mlp_train}


# ---- inputs ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = TORCH_DTYPES[case["dtype"]] if "dtype" in case else torch.bfloat16

    def normal(*shape, std=1.0, mean=0.0):
        return (torch.randn(shape, generator=gen, device="cuda") * std + mean).to(dtype)

    kind, state = case["kind"], {"case": dict(case)}
    if kind == "chain":
        rows, cols = case["rows"], case["cols"]
        g = (torch.rand(cols, generator=gen, device="cuda") + 0.5).to(dtype)
        state["args"] = [normal(rows, cols), g, normal(cols, std=0.1)]
    elif kind == "norm":
        rows, cols = case["rows"], case["cols"]
        state["args"] = [normal(rows, cols), normal(rows, cols), normal(cols, std=0.1, mean=1.0), normal(cols, std=0.1), normal(rows, cols)]
    elif kind == "mlp":
        t, d, h = case["tokens"], case["width"], case["hidden"]
        state["args"] = [normal(t, d), normal(d, h, std=d**-0.5), normal(h, d, std=h**-0.5), normal(t, d)]
    elif kind == "matmul":
        m, n, k = case["m"], case["n"], case["k"]
        state["a"], state["b"], state["dy"] = normal(m, k, std=k**-0.5), normal(k, n, std=k**-0.5), normal(m, n)
        state["y"] = torch.empty((m, n), dtype=torch.float32, device="cuda")
        state["da"], state["db"] = torch.empty_like(state["a"]), torch.empty_like(state["b"])
    elif kind == "attention":
        b, sq, sk, d = case["batch"], case["queries"], case["keys"], case["dim"]
        state["q"] = normal(b, sq, case["heads"], d)
        state["k"], state["v"] = normal(b, sk, case["kv_heads"], d), normal(b, sk, case["kv_heads"], d)
        if case["backward"]:
            state["d_o"] = normal(b, sq, case["heads"], d)
    else:
        cfg = transformer.Config(vocab=case["vocab"], d_model=case["width"], heads=case["heads"], hidden=case["hidden"],
                                 layers=case["layers"], seq=case["seq"], dtype=case["dtype"], logits_dtype=case["dtype"],
                                 optimizer=case["optimizer"], lr=1e-2 if case["optimizer"] == "sgd" else 1e-3)
        # weights N(0, 0.02), layer-norm scales and biases around 1 and 0 as after some training
        params = {}
        for name, shape in transformer.param_shapes(cfg):
            w = (normal(*shape, std=0.1, mean=1.0) if name.endswith("norm.w") else
                 normal(*shape, std=0.1) if name.endswith("norm.b") else normal(*shape, std=0.02))
            params[name] = _host(w)
        step = transformer.TrainStep(cfg, case["batch"], params, torch.cuda.current_device(), deterministic=case["deterministic"])
        tokens = torch.randint(0, cfg.vocab, (case["batch"], cfg.seq + 1), generator=gen, device="cuda").cpu()
        state["ids"], state["targets"] = tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous()
        step.load_batch(state["ids"], state["targets"])
        step.synchronize()
        state["step"] = step
        state["outputs"] = [_on_torch(t) for t in (step.loss, *step.params, *step.moments)]
    return state


def _host(t):
    """A GPU tensor's values as the NumPy array a checkpoint gives: bfloat16 by its bit pattern."""
    if t.dtype != torch.bfloat16:
        return t.cpu().numpy()
    import ml_dtypes

    return t.cpu().view(torch.int16).numpy().view(ml_dtypes.bfloat16)


def _on_torch(t):
    """The memory of one of the backend's tensors as a torch tensor."""
    if t.dtype == "bfloat16":
        return torch.as_tensor(t, device="cuda").view(torch.bfloat16)
    return torch.as_tensor(t, device="cuda")


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in PROGRAMS:
        return compiled(PROGRAMS[kind])(*state["args"])
    if kind == "matmul":
        a, b, dy = state["a"], state["b"], state["dy"]
        runtime.gemm(a, b, state["y"])
        runtime.gemm(dy, b.t(), state["da"])
        runtime.gemm(a.t(), dy, state["db"])
        return state["y"], state["da"], state["db"]
    if kind == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        o, lse = runtime.attention_forward(q, k, v, causal=case["causal"])
        if not case["backward"]:
            return o, lse
        grads = runtime.attention_backward(q, k, v, o, state["d_o"], lse, causal=case["causal"], deterministic=case["deterministic"])
        return (o, lse, *grads)
    state["step"].step()
    return state["outputs"]


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "chain":
        n, c, e = case["rows"] * case["cols"], case["cols"], ITEM[case["dtype"]]
        return {"bytes": 2 * n * e + 2 * c * e + 4 * case["rows"], "flops": 5 * n}
    if kind == "norm":
        n, c, e = case["rows"] * case["cols"], case["cols"], ITEM[case["dtype"]]
        return {"bytes": 5 * n * e + 4 * c * e, "flops": 25 * n}  # x, r, dy read; y, dx written; w, b, dw, db
    if kind == "mlp":
        t, d, h, e = case["tokens"], case["width"], case["hidden"], ITEM[case["dtype"]]
        return {"bytes": (4 * t * d + 4 * d * h) * e, "flops": 12 * t * d * h}
    if kind == "matmul":
        m, n, k, e = case["m"], case["n"], case["k"], ITEM[case["dtype"]]
        return {"bytes": (2 * m * k + 2 * k * n + m * n) * e + 4 * m * n, "flops": 6 * m * n * k}
    if kind == "attention":
        b, n, nkv, sq, sk, d = case["batch"], case["heads"], case["kv_heads"], case["queries"], case["keys"], case["dim"]
        pairs = sq * sk - sq * (sq - 1) // 2 if case["causal"] else sq * sk
        q, kv, rows = 2 * b * sq * n * d, 2 * b * sk * nkv * d, 4 * b * n * sq
        if case["backward"]:  # q, k, v, dO read; o, lse, dq, dk, dv written
            return {"bytes": 4 * q + 4 * kv + rows, "flops": 14 * b * n * pairs * d}
        return {"bytes": 2 * q + 2 * kv + rows, "flops": 4 * b * n * pairs * d}
    cfg = transformer.Config(vocab=case["vocab"], d_model=case["width"], heads=case["heads"], hidden=case["hidden"], layers=case["layers"],
                             seq=case["seq"])
    weights = sum(int(np.prod(shape)) for _, shape in transformer.param_shapes(cfg))
    state = weights * ITEM[case["dtype"]] + (8 * weights if case["optimizer"] == "adamw" else 0)
    return {"bytes": 2 * state + 16 * case["batch"] * case["seq"], "flops": transformer.flops_per_step(cfg, case["batch"])}


def tolerance(case):
    if case["kind"] == "step" and case["dtype"] == "float32":
        return {"rel": 1e-4}  # gradients are sums over all tokens through every layer; the parity tests hold them to this
    if case.get("dtype", "bfloat16") == "float32":
        return {"rel": 1e-5}
    return {"rel": 1e-2}  # one 16-bit rounding of each result, of probabilities and of activations on the way
