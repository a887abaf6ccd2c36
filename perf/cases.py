"""The work this library is called for, as cases that a timing harness can run.

A case is a dict of plain values.  `kind` says which public entry points it goes through:

    linear      mlx_b200.quantized_matmul(x, w, scales, biases): one linear layer of a model whose weights are
                quantized, M token rows at once (M = 1: one sequence being decoded, up to 16: a small batch of
                them, above: prompts and large batches)
    train       mlx_b200.grad.quantized_matmul and its backward pass with respect to x: the frozen quantized
                layer under a low-rank adapter that is being fine-tuned
    experts     mlx_b200.gather_qmm: one projection of a mixture-of-experts layer, `top` experts per token
    expert_mlp  mlx_b200.gather_qmm_swiglu: the whole gated expert layer, for the few tokens of a decode step
    convert     mlx_b200.quantize and mlx_b200.dequantize of one weight matrix: a checkpoint being converted
                and checked

Activations are N(0, 1) and weights N(0, 0.02), as they are in the benchmark configurations of this repository;
routing draws `top` different experts per token uniformly.
"""
import math

import torch

import mlx_b200
from mlx_b200 import grad

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _linear(M, N, K, bits, group, dtype):
    return {"kind": "linear", "M": M, "N": N, "K": K, "bits": bits, "group": group, "dtype": dtype}


def _train(M, N, K, bits, group, dtype):
    return {"kind": "train", "M": M, "N": N, "K": K, "bits": bits, "group": group, "dtype": dtype}


def _experts(kind, tokens, E, top, N, K, bits, group):
    return {"kind": kind, "tokens": tokens, "E": E, "top": top, "N": N, "K": K, "bits": bits, "group": group, "dtype": "bf16"}


def _convert(N, K, bits, group, dtype):
    return {"kind": "convert", "N": N, "K": K, "bits": bits, "group": group, "dtype": dtype}


def listed():
    return [
        # one token through a square attention projection: the smallest call a decode loop makes
        {"name": "decode 1 row", **_linear(1, 4096, 4096, 4, 64, "bf16")},
        # sixteen sequences decoded together through an MLP up-projection: the benchmark's default workload
        {"name": "decode 16 rows", **_linear(16, 14336, 4096, 4, 64, "bf16")},
        # one token through the widest MLP matrix, at a field width that straddles bytes
        {"name": "decode wide 6-bit", **_linear(1, 28672, 8192, 6, 32, "bf16")},
        # a model kept in half precision with 8-bit weights, three sequences
        {"name": "decode f16 8-bit", **_linear(3, 11008, 4096, 8, 64, "f16")},
        # a short prompt, or a server's batch, through a down-projection: neither decode nor a full tile
        {"name": "batch 57 rows", **_linear(57, 4096, 11008, 4, 64, "bf16")},
        # a long prompt: the dense tensor-core case
        {"name": "prefill 4096", **_linear(4096, 14336, 4096, 4, 64, "bf16")},
        # a chunk of a prompt through the widest MLP matrix at 3 bits
        {"name": "prefill 512 3-bit", **_linear(512, 28672, 8192, 3, 128, "bf16")},
        # a prompt of odd length on a half-precision model
        {"name": "prefill f16", **_linear(1531, 14336, 4096, 4, 64, "f16")},
        # fine-tuning: 1024 tokens forward and backward through a frozen layer
        {"name": "train 1024", **_train(1024, 14336, 4096, 4, 64, "bf16")},
        # 512 tokens, top-2 of 8 experts: a prompt through a mixture-of-experts projection
        {"name": "experts 512 tokens", **_experts("experts", 512, 8, 2, 14336, 4096, 4, 64)},
        # four sequences decoded together through the gated experts
        {"name": "expert mlp 4 tokens", **_experts("expert_mlp", 4, 8, 2, 14336, 4096, 4, 64)},
        # the widest matrix of a checkpoint, quantized and read back
        {"name": "convert", **_convert(28672, 8192, 4, 64, "bf16")},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo=1024, hi=28672):
    """A layer's input or output width: whole blocks of 256."""
    return max(lo, _log_int(rng, lo, hi) // 256 * 256)


def _matrix(rng, most=28672 * 8192):
    while True:
        N, K = _width(rng), _width(rng)
        if N * K <= most:
            return N, K


def draw(rng):
    bits = rng.choice((2, 3, 4, 4, 4, 4, 5, 6, 8, 8))
    group = rng.choice((32, 64, 64, 128))
    dtype = rng.choice(("bf16", "bf16", "f16"))
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "train", "experts", "expert_mlp", "convert"))
    if kind in ("decode", "prefill"):
        N, K = _matrix(rng)
        if rng.random() < 0.25:   # an output head: vocabularies come in any size
            N -= rng.randrange(1, 64)
        # no more work than a long prompt has; in half precision no more than the listed half-precision prompt
        most = (4096 if dtype == "bf16" else 1531) * 14336 * 4096
        M = _log_int(rng, 1, 16) if kind == "decode" else _log_int(rng, 17, min(4096, most // (N * K)))
        return _linear(M, N, K, bits, group, dtype)
    if kind == "train":
        N, K = _matrix(rng, 14336 * 4096)
        return _train(_log_int(rng, 128, min(4096, 1024 * 14336 * 4096 // (N * K))), N, K, bits, group, dtype)
    if kind == "experts":
        E = rng.choice((4, 8, 16, 32, 64))
        top = rng.choice((1, 2, 4))
        N, K = _matrix(rng, 8 * 14336 * 4096 // E)
        return _experts(kind, _log_int(rng, 16, 1024 // top), E, top, N, K, bits, group)
    if kind == "expert_mlp":
        E = rng.choice((4, 8, 16, 32, 64))
        top = rng.choice((1, 2, 4))
        N, K = _matrix(rng, 8 * 14336 * 4096 // E)
        return _experts(kind, _log_int(rng, 1, 16), E, top, N, K, bits, group)
    N, K = _matrix(rng)
    dtype = rng.choice(("bf16", "f16", "f32"))
    if dtype == "f32":
        N = max(1, N // 2)
    return _convert(N - rng.choice((0, 0, rng.randrange(1, 64))), K, bits, group, dtype)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, shape, dtype, std=1.0):
    t = torch.randn(shape, generator=g, device="cuda", dtype=dtype)
    return t if std == 1.0 else t.mul_(std)


def prepare(case, seed):
    g, c = _gen(seed), case
    dt = _DTYPES[c["dtype"]]
    q = {"group_size": c["group"], "bits": c["bits"]}
    if c["kind"] == "convert":
        return {"kind": "convert", "w": _normal(g, (c["N"], c["K"]), dt, 0.02), "q": q}
    if c["kind"] in ("linear", "train"):
        w = mlx_b200.quantize(_normal(g, (c["N"], c["K"]), dt, 0.02), **q)
        s = {"kind": c["kind"], "w": w, "q": q, "x": _normal(g, (c["M"], c["K"]), dt)}
        if c["kind"] == "train":
            s["x"].requires_grad_(True)
            s["dy"] = _normal(g, (c["M"], c["N"]), dt)
        return s
    E, N, K = c["E"], c["N"], c["K"]
    s = {"kind": c["kind"], "q": q, "x": _normal(g, (c["tokens"], 1, 1, K), dt)}
    s["idx"] = torch.rand((c["tokens"], E), generator=g, device="cuda").topk(c["top"], dim=-1).indices
    if c["kind"] == "experts":
        s["w"] = mlx_b200.quantize(_normal(g, (E, N, K), dt, 0.02), **q)
    else:
        s["gate"] = mlx_b200.quantize(_normal(g, (E, N, K), dt, 0.02), **q)
        s["up"] = mlx_b200.quantize(_normal(g, (E, N, K), dt, 0.02), **q)
        s["down"] = mlx_b200.quantize(_normal(g, (E, K, N), dt, 0.02), **q)
    return s


def run(s):
    kind, q = s["kind"], s["q"]
    if kind == "linear":
        return mlx_b200.quantized_matmul(s["x"], *s["w"], **q)
    if kind == "train":
        y = grad.quantized_matmul(s["x"], *s["w"], **q)
        return y, torch.autograd.grad(y, s["x"], s["dy"])[0]
    if kind == "experts":
        return mlx_b200.gather_qmm(s["x"], *s["w"], rhs_indices=s["idx"], **q)
    if kind == "expert_mlp":
        return mlx_b200.gather_qmm_swiglu(s["x"], s["gate"], s["up"], s["down"], s["idx"], **q)
    wq, scales, biases = mlx_b200.quantize(s["w"], **q)
    return wq.view(torch.int32), scales, biases, mlx_b200.dequantize(wq, scales, biases, **q)


def _packed(N, K, c):
    """Bytes of a quantized N x K matrix: fields, and a scale and a bias per group."""
    return N * K * c["bits"] / 8 + 2 * (N * K // c["group"]) * (4 if c["dtype"] == "f32" else 2)


def work(case):
    c = case
    N, K = c["N"], c["K"]
    size = 4 if c["dtype"] == "f32" else 2
    if c["kind"] == "convert":   # read w; write the packed form and read it again; write the values
        return {"bytes": 2 * N * K * size + 2 * _packed(N, K, c), "flops": 0}
    if c["kind"] in ("linear", "train"):
        M = c["M"]
        b, f = _packed(N, K, c) + M * K * size + M * N * size, 2 * M * N * K
        if c["kind"] == "train":   # the weights once more, dy read, dx written
            return {"bytes": 2 * b, "flops": 2 * f}
        return {"bytes": b, "flops": f}
    # the expected number of different experts that a draw of `top` per token reaches
    rows = c["tokens"] * c["top"]
    used = c["E"] * (1 - (1 - c["top"] / c["E"]) ** c["tokens"])
    b, f = used * _packed(N, K, c) + c["tokens"] * K * size, 2 * rows * N * K
    if c["kind"] == "experts":
        return {"bytes": b + rows * N * size, "flops": f}
    return {"bytes": 3 * used * _packed(N, K, c) + (c["tokens"] + rows) * K * size, "flops": 3 * f}


def tolerance(case):
    if case["kind"] == "convert":
        return "exact"   # the packed fields, scales and biases are defined bit for bit, and so are the values
    if case["dtype"] == "f16":
        return {"rel": 2e-3, "max": 0.02}
    # bf16: the weights' and the result's rounding, 2^-9 each
    return {"rel": 1e-2, "max": 0.1}
