"""What users of this framework have it do, as cases that can be timed: products of a block-sparse weight with
activations in every element type, the linear layers and the training step built on them, and the conversion of a
pruned dense weight.  Sizes are those of the repository's workloads (512^2, 4096^2, 16384^2 and 65536^2 block-sparse
matrices of 32x32 tiles) and generic layer widths; ``draw`` spreads over the ranges between them, ragged sizes included.

A case is a dict of plain values; ``op`` says which path it takes:
  spmv     y = A x, floating point                                            void_spmv
  int8     C = dequant(A_q B_q), fp16 result; quant_b: the activations arrive in fp32 and are quantised
           per column in the same pass                                        quantize_cols_int8, void_spmm_int8
  fp8      the same in E4M3                                                   quantize_cols_fp8, void_spmm_fp8
  fp       C = A B in fp32 (TF32 products), fp16 or bf16; act: fused GELU with a column bias
                                                                              void_spmm, void_spmm_gelu
  streamk  A with power-law tile-row lengths, INT8, split by the work plan, fused GELU, bf16 result
                                                                              void_spmm_stream_k
  mlp      two sparse linear layers with biases and GELU, inference           fused_sparse_mlp
  train    one training step of a sparse linear layer: forward, gradients of input, tiles and bias, and the
           update of the parameters                                           SparseLinear
  convert  a pruned dense weight becomes a quantised VOID tensor and serves its first product
                                                         dense_to_void, quantize_void_tensor, void_spmm_int8
"""
import math

import torch

import void_b200 as void
from void_b200 import workloads

TILE = 32
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
GELU = void.get_activation_code("gelu")
LEARNING_RATE = 1e-5
LARGEST_OPS = 4.6e11     # multiply-adds x 2 of the largest listed case
LARGEST_BYTES = 4.3e8    # and its bytes


def listed():
    return [
        # the smallest call: one matrix-vector product with the 512^2 plumbing matrix, whose tiles are all stored
        {"name": "spmv_512", "op": "spmv", "m": 512, "k": 512, "n": 1, "sparsity": 0.0, "dtype": "fp32"},
        # the plumbing workload in INT8, activations quantised on the way: a small layer in a served network
        {"name": "int8_512_dynamic", "op": "int8", "m": 512, "k": 512, "n": 128, "sparsity": 0.0, "quant_b": True},
        # the headline workload: INT8, 90 % block sparsity, activations already quantised
        {"name": "int8_4096", "op": "int8", "m": 4096, "k": 4096, "n": 512, "sparsity": 0.9, "quant_b": False},
        # one point of the FP8 sparsity sweep, activations quantised on the way
        {"name": "fp8_4096_dynamic", "op": "fp8", "m": 4096, "k": 4096, "n": 512, "sparsity": 0.8, "quant_b": True},
        # the same sweep in fp32, the configuration of the published timings
        {"name": "fp32_4096", "op": "fp", "m": 4096, "k": 4096, "n": 512, "sparsity": 0.9, "dtype": "fp32", "act": False},
        # sizes that are multiples of nothing: edges of tiles, panels and the copy engine's 16 bytes
        {"name": "bf16_gelu_ragged", "op": "fp", "m": 3001, "k": 5003, "n": 333, "sparsity": 0.85, "dtype": "bf16",
         "act": True},
        # power-law rows under the balanced work plan with fused GELU
        {"name": "int8_streamk_16384", "op": "streamk", "m": 16384, "k": 16384, "n": 256},
        # generation: a handful of tokens through two sparse layers
        {"name": "mlp_decode", "op": "mlp", "k": 2048, "m": 8192, "n": 8, "sparsity": 0.8, "dtype": "fp16"},
        # prompt processing: a few thousand tokens through wider layers
        {"name": "mlp_prefill", "op": "mlp", "k": 4096, "m": 16384, "n": 2048, "sparsity": 0.9, "dtype": "bf16"},
        # a training step at the size of the published sweep
        {"name": "train_4096", "op": "train", "m": 4096, "k": 4096, "n": 512, "sparsity": 0.9, "dtype": "fp32"},
        # loading a pruned layer: dense weight to quantised tiles to the first product
        {"name": "convert_4096", "op": "convert", "m": 4096, "k": 4096, "n": 512, "sparsity": 0.8, "dtype": "fp32"},
        # the largest: the scaling workload on one GPU
        {"name": "int8_65536", "op": "int8", "m": 65536, "k": 65536, "n": 1024, "sparsity": 0.95, "quant_b": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _side(rng, lo, hi):
    """A matrix side over the whole range: a multiple of 128, a multiple of the tile, or any number."""
    v = _log_int(rng, lo, hi)
    unit = rng.choice((128, 32, 1))
    return max(lo, v // unit * unit)


def _columns(rng, lo, hi):
    v = _log_int(rng, lo, hi)
    unit = rng.choice((64, 8, 1))
    return max(lo, v // unit * unit)


def draw(rng):
    while True:
        op = rng.choice(("spmv", "int8", "int8", "fp8", "fp", "fp", "streamk", "mlp", "mlp", "train", "convert"))
        sparsity = round(rng.uniform(0.5, 0.98), 3)
        dtype = rng.choice(("fp32", "fp16", "bf16"))
        if op == "spmv":
            c = {"op": op, "m": _side(rng, 256, 16384), "k": _side(rng, 256, 16384), "n": 1, "sparsity": sparsity,
                 "dtype": dtype}
        elif op in ("int8", "fp8"):
            top = 65536 if op == "int8" else 16384
            c = {"op": op, "m": _side(rng, 256, top), "k": _side(rng, 256, top), "n": _columns(rng, 8, 2048),
                 "sparsity": sparsity, "quant_b": rng.random() < 0.5}
        elif op == "fp":
            c = {"op": op, "m": _side(rng, 256, 16384), "k": _side(rng, 256, 16384), "n": _columns(rng, 8, 2048),
                 "sparsity": sparsity, "dtype": dtype, "act": rng.random() < 0.5}
        elif op == "streamk":
            c = {"op": op, "m": _side(rng, 2048, 32768), "k": _side(rng, 2048, 32768), "n": _columns(rng, 32, 1024)}
        elif op == "mlp":
            c = {"op": op, "k": _side(rng, 512, 8192), "m": _side(rng, 512, 16384), "n": _columns(rng, 1, 4096),
                 "sparsity": sparsity, "dtype": rng.choice(("fp16", "bf16"))}
        elif op == "train":
            c = {"op": op, "m": _side(rng, 256, 8192), "k": _side(rng, 256, 8192), "n": _columns(rng, 16, 4096),
                 "sparsity": sparsity, "dtype": rng.choice(("fp32", "bf16"))}
        else:
            c = {"op": op, "m": _side(rng, 256, 8192), "k": _side(rng, 256, 8192), "n": _columns(rng, 16, 1024),
                 "sparsity": sparsity, "dtype": rng.choice(("fp32", "bf16"))}
        w = work(c)
        # tensor-core work counts by element size, so that no drawn case takes longer than the largest listed one
        if w["flops"] * _elem_bytes(c) <= LARGEST_OPS and w["bytes"] <= LARGEST_BYTES:
            return c


def _elem_bytes(c):
    return {"fp32": 4, "fp16": 2, "bf16": 2}.get(c.get("dtype"), 1)


# ------------------------------------------------------------------------------------------ inputs
def _side_tiles(side):
    return (side + TILE - 1) // TILE


def _stored_tiles(case):
    """Number of stored tiles of A (the expected number for power-law rows)."""
    cells = _side_tiles(case["m"]) * _side_tiles(case["k"])
    if case["op"] == "streamk":
        return 0.03 * cells
    return max(1, round((1.0 - case["sparsity"]) * cells))


def _mask(gen, nbr, nbc, count):
    """Block mask with ``count`` stored tiles at uniformly random places."""
    mask = torch.zeros(nbr * nbc, dtype=torch.bool, device="cuda")
    mask[torch.rand(nbr * nbc, generator=gen, device="cuda").argsort()[:count]] = True
    return mask.view(nbr, nbc)


def _block_sparse(gen, m, k, mask, dtype=torch.float32, scale=1.0):
    """VOIDTensor with N(0, scale) tiles on the block mask, zero outside the matrix like every converted one."""
    values = torch.randn(int(mask.sum()), TILE, TILE, generator=gen, device="cuda") * scale
    a = void.void_from_block_mask(mask.cpu().numpy(), values, shape=(m, k))
    if m % TILE:
        a.values[a.block_rows == m // TILE, m % TILE:, :] = 0
    if k % TILE:
        a.values[a.block_cols == k // TILE, :, k % TILE:] = 0
    return a if dtype == torch.float32 else a.to_dtype(dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op, m, k, n = case["op"], case["m"], case["k"], case["n"]
    dtype = DTYPES[case.get("dtype", "fp32")]
    nbr, nbc = _side_tiles(m), _side_tiles(k)
    stored = _stored_tiles(case)

    def randn(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device="cuda").to(dtype)

    s = {"case": dict(case)}
    if op == "spmv":
        s["a"] = _block_sparse(gen, m, k, _mask(gen, nbr, nbc, stored), dtype)
        s["x"] = randn(k, dtype=dtype)
    elif op in ("int8", "fp8"):
        a = _block_sparse(gen, m, k, _mask(gen, nbr, nbc, stored))
        s["a"] = void.quantize_void_tensor(a) if op == "int8" else void.void_tensor_to_fp8(a)
        b = randn(k, n)
        if case["quant_b"]:
            s["b"] = b
        elif op == "int8":
            s["b"], s["b_scale"] = void.quantize_cols_int8(b)
        else:
            s["b"], s["b_scale"], _ = void.quantize_cols_fp8(b)
    elif op == "fp":
        s["a"] = _block_sparse(gen, m, k, _mask(gen, nbr, nbc, stored), dtype)
        s["b"] = randn(k, n, dtype=dtype)
        s["bias"] = randn(n) if case["act"] else None
    elif op == "streamk":
        mask = torch.from_numpy(workloads.zipf_mask(nbr, nbc, 1.5, 512, 0.03 * nbc, int(seed)))
        s["a"] = void.quantize_void_tensor(_block_sparse(gen, m, k, mask))
        s["b"], s["b_scale"] = void.quantize_cols_int8(randn(k, n))
    elif op == "mlp":
        kept = 1.0 - case["sparsity"]
        s["w1"] = _block_sparse(gen, m, k, _mask(gen, nbr, nbc, stored), dtype, (kept * k) ** -0.5)
        s["w2"] = _block_sparse(gen, k, m, _mask(gen, nbc, nbr, stored), dtype, (kept * m) ** -0.5)
        s["b1"], s["b2"] = randn(m), randn(k)
        s["x"] = randn(n, k, dtype=dtype)
    elif op == "train":
        a = _block_sparse(gen, m, k, _mask(gen, nbr, nbc, stored), dtype, ((1.0 - case["sparsity"]) * k) ** -0.5)
        s["layer"] = void.SparseLinear(k, m, a, bias=True)
        s["x"] = randn(n, k, dtype=dtype).requires_grad_(True)
        s["grad"] = randn(n, m, dtype=dtype) / n
    else:
        mask = _mask(gen, nbr, nbc, stored)
        w = randn(m, k) * mask.repeat_interleave(TILE, 0).repeat_interleave(TILE, 1)[:m, :k]
        s["w"] = w.to(dtype)
        s["b"], s["b_scale"] = void.quantize_cols_int8(randn(k, n))
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "spmv":
        return void.void_spmv(s["a"], s["x"])
    if op == "int8":
        b, scale = void.quantize_cols_int8(s["b"]) if case["quant_b"] else (s["b"], s["b_scale"])
        return void.void_spmm_int8(s["a"], b, scale, out_dtype=torch.float16)
    if op == "fp8":
        b, scale = void.quantize_cols_fp8(s["b"])[:2] if case["quant_b"] else (s["b"], s["b_scale"])
        return void.void_spmm_fp8(s["a"], b, torch.float16, b_scale=scale)
    if op == "fp":
        if case["act"]:
            return void.void_spmm_gelu(s["a"], s["b"], s["bias"])
        return void.void_spmm(s["a"], s["b"])
    if op == "streamk":
        return void.void_spmm_stream_k(s["a"], s["b"], b_scale=s["b_scale"], out_dtype=torch.bfloat16, activation=GELU)
    if op == "mlp":
        return void.fused_sparse_mlp(s["x"], s["w1"], s["w2"], "gelu", s["b1"], s["b2"])
    if op == "train":
        layer, x = s["layer"], s["x"]
        params = list(layer.parameters())
        for p in params:
            p.grad = None
        x.grad = None
        y = layer(x)
        y.backward(s["grad"])
        with torch.no_grad():
            for p in params:
                p.add_(p.grad, alpha=-LEARNING_RATE)
        return {"y": y.detach(), "dx": x.grad, "grads": [p.grad for p in params], "params": [p.detach() for p in params]}
    a = void.dense_to_void(s["w"])
    q = void.quantize_void_tensor(a)
    c = void.void_spmm_int8(q, s["b"], s["b_scale"], out_dtype=torch.float16)
    return {"values": q.values, "scales": q.scales, "block_rows": q.block_rows, "block_cols": q.block_cols,
            "morton_codes": a.morton_codes, "c": c}


# ------------------------------------------------------------------------------------------ what a pass is worth
def work(case):
    """Bytes and operations of one pass: every stored tile with its index (and scale), the dense operand and the
    result once each; two operations per multiply-add over the stored tiles."""
    op, m, k, n = case["op"], case["m"], case["k"], case["n"]
    es = _elem_bytes(case)
    tiles = _stored_tiles(case)
    index = 4 * (_side_tiles(m) + 1)
    ops = 2.0 * tiles * TILE * TILE * n
    if op in ("int8", "fp8"):
        b = k * n * 4 if case["quant_b"] else k * n + 4 * n
        return {"bytes": tiles * 1032 + index + b + 2 * m * n, "flops": ops}
    if op == "streamk":
        return {"bytes": tiles * 1032 + index + k * n + 4 * n + 2 * m * n, "flops": ops}
    if op in ("spmv", "fp"):
        return {"bytes": tiles * (1024 * es + 4) + index + es * (k * n + m * n), "flops": ops}
    if op == "mlp":
        # both weights, x in and y out
        return {"bytes": 2 * (tiles * (1024 * es + 4) + index) + es * n * 2 * k, "flops": 2 * ops}
    if op == "train":
        # tiles, x and dL/dy in; y, both gradients and the updated tiles out
        return {"bytes": tiles * (3 * 1024 * es + 4) + index + es * n * 2 * (k + m), "flops": 3 * ops}
    # the dense weight and the activations in; quantised tiles with scales and coordinates, and the product out
    return {"bytes": es * m * k + tiles * 1044 + k * n + 4 * n + 2 * m * n, "flops": ops}


def tolerance(case):
    op, dtype = case["op"], case.get("dtype", "fp32")
    if op in ("int8", "convert"):
        return {"rel": 1e-3}            # int32 sums are exact, the result is rounded to fp16; whole values are the same
    if op == "streamk":
        return {"rel": 5e-3}            # exact sums, hardware exp in GELU, bf16 result
    if op == "fp8":
        return {"rel": 3e-3}            # A with its tile scale in 8 significant bits, fp32 sums, fp16 result
    if dtype == "bf16":
        return {"rel": 1e-2}
    if dtype == "fp16":
        return {"rel": 2e-3}
    return {"rel": 1e-3}                # fp32 operands multiplied as TF32
