"""The workloads this library is measured on: ternary products and the blocks built from them, through the calls that a
user's program makes, over the sizes, row counts, data types and layouts it is used with.

A case names a `kind`, which says what is called:

  linear   PackedWeight.matmul on a packed weight, device tensors (decode and prefill projections, int8 included)
  host     PackedWeight.matmul_host: host arrays in and out (the calling convention of the CPU kernel entry points)
  lists    ter_spmm.ter_spmm on the merged tiled CSC arrays as they are (code written against the three buffers)
  mlp      PackedMLP.forward: gate, up, SiLU * mul, down of one block
  module   LlamaTernaryMLP.forward, the module form
  attn     LlamaTernaryAttention.forward, causal, no cache: q | k | v and o projections around the stock attention core
  layer    one decode step of TernaryDecoderLayerTP on one GPU, replayed from a CUDA graph as a serving loop does

Sizes are those of the repository's configurations and benchmark: hidden 2048 / FFN 8192 (32 and 8 heads of 64), 4096 /
11008, 5120 / 15360 and 8192 / 10240.  `zeros` is the share of zero entries in W.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ternaryllm_b200 import LlamaTernaryAttention, LlamaTernaryMLP, PackedMLP, PackedWeight, TernaryConfig, TernaryDecoderLayerTP, ter_spmm

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i8": torch.int8}
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "i8": 1}
SCALE = 0.03125
KV_LEN = 1024                 # cached positions of the decode step
MAX_ENTRIES = 5120 * 15360    # of one weight


def listed():
    return [
        # one small fp32 product on eight rows: the single-GEMM configuration, where launches and host time count
        {"name": "linear f32 m8 2048x2048", "kind": "linear", "dtype": "f32", "M": 8, "K": 2048, "N": 2048, "zeros": 0.5},
        # one token through the up-projection of a 4096-wide model
        {"name": "linear f16 m1 4096x11008", "kind": "linear", "dtype": "f16", "M": 1, "K": 4096, "N": 11008, "zeros": 0.75},
        # one token through the fused QKV projection of an 8192-wide model
        {"name": "linear bf16 m1 8192x10240", "kind": "linear", "dtype": "bf16", "M": 1, "K": 8192, "N": 10240, "zeros": 0.5},
        # a projection whose sizes are multiples of nothing: rows of X that start on odd addresses, ragged tiles
        {"name": "linear bf16 m3 1003x517", "kind": "linear", "dtype": "bf16", "M": 3, "K": 1003, "N": 517, "zeros": 0.6},
        # quantised activations, exact integer sums
        {"name": "linear i8 m32 2048x8192", "kind": "linear", "dtype": "i8", "M": 32, "K": 2048, "N": 8192, "zeros": 0.5},
        # prefill of the QKV projection of a 5120-wide model
        {"name": "linear bf16 m2048 5120x15360", "kind": "linear", "dtype": "bf16", "M": 2048, "K": 5120, "N": 15360, "zeros": 0.5},
        # host buffers in the column-major layout of the CPU kernels, at the row count of their prefill benchmark
        {"name": "host f32 m256 1024x4096", "kind": "host", "dtype": "f32", "M": 256, "K": 1024, "N": 4096, "zeros": 0.7, "col_major": True},
        # 256 positions on the index arrays as they are
        {"name": "lists f32 m256 2048x8192", "kind": "lists", "dtype": "f32", "M": 256, "K": 2048, "N": 8192, "zeros": 0.8},
        # the fused MLP block of a 4096-wide model on a decode batch
        {"name": "mlp f16 m8 4096x11008", "kind": "mlp", "dtype": "f16", "M": 8, "K": 4096, "N": 11008, "zeros": 0.6},
        # the MLP and attention modules on 256 positions in fp32
        {"name": "module f32 m256 2048x8192", "kind": "module", "dtype": "f32", "M": 256, "K": 2048, "N": 8192, "zeros": 0.8},
        {"name": "attn f32 m256 2048", "kind": "attn", "dtype": "f32", "M": 256, "K": 2048, "N": 2048, "heads": 32, "kv_heads": 8, "zeros": 0.8},
        # one decode step of a whole layer, batch 16
        {"name": "layer bf16 m16 2048x8192", "kind": "layer", "dtype": "bf16", "M": 16, "K": 2048, "N": 8192, "heads": 32, "kv_heads": 8, "zeros": 0.5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm: one in three as it comes (mostly odd), the others rounded to
    a multiple of 8, 64 or 128, as the sizes of models are."""
    v = _log(rng, lo, hi)
    step = rng.choice((1, 1, 8, 64, 128, 128))
    return min(hi, max(lo, (v + step // 2) // step * step))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "linear", "linear", "host", "lists", "mlp", "module", "attn", "layer"))
    zeros = rng.choice((0.5, 0.6, 0.7, 0.75, 0.8, 0.9))
    if kind == "linear":
        K, N = _size(rng, 256, 8192), _size(rng, 256, 15360)
        while K * N > MAX_ENTRIES // 2:
            K, N = _size(rng, 256, 8192), _size(rng, 256, 15360)
        return {"kind": kind, "dtype": rng.choice(("f32", "f16", "f16", "bf16", "bf16", "i8")), "M": _log(rng, 1, 2048), "K": K, "N": N, "zeros": zeros}
    if kind == "host":
        return {"kind": kind, "dtype": rng.choice(("f32", "f32", "f16", "i8")), "M": _log(rng, 1, 256), "K": _size(rng, 256, 2048),
                "N": _size(rng, 256, 8192), "zeros": zeros, "col_major": rng.choice((True, False))}
    if kind == "lists":
        return {"kind": kind, "dtype": rng.choice(("f32", "f32", "f16", "bf16")), "M": _log(rng, 1, 256), "K": _size(rng, 256, 2048),
                "N": _size(rng, 256, 8192), "zeros": zeros}
    if kind in ("mlp", "module"):
        return {"kind": kind, "dtype": rng.choice(("f32", "f16", "bf16")), "M": _log(rng, 1, 512), "K": _size(rng, 256, 2560),
                "N": _size(rng, 512, 6912), "zeros": zeros}
    hd = rng.choice((64, 128))
    groups = rng.choice((1, 4))
    if kind == "attn":
        heads = 4 * rng.randint(2, 2048 // (4 * hd))
        return {"kind": kind, "dtype": rng.choice(("f32", "f16", "bf16")), "M": _log(rng, 16, 512), "K": heads * hd, "N": heads * hd, "heads": heads,
                "kv_heads": heads // groups, "zeros": zeros}
    heads = 8 * rng.randint(1, 2048 // (8 * hd))
    kv = heads // groups if heads // groups % 8 == 0 else 8
    return {"kind": kind, "dtype": "bf16", "M": _log(rng, 1, 64), "K": heads * hd, "N": 128 * rng.randint(8, 64), "heads": heads, "kv_heads": kv,
            "zeros": zeros}


def _ternary(gen, K, N, zeros):
    """Seeded ternary matrix [K, N] on the host: i.i.d. zeros with the given probability, +1 and -1 equiprobable."""
    z = int(round(zeros * 256))
    half = (256 - z) // 2
    r = torch.randint(0, 256, (K, N), dtype=torch.uint8, device="cuda", generator=gen)
    w = (r >= z + half).to(torch.int8) - ((r >= z) & (r < z + half)).to(torch.int8)
    return w.cpu().numpy()


def _activations(gen, shape, dtype):
    if dtype == "i8":
        return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=gen)
    return torch.randn(shape, device="cuda", generator=gen).to(DTYPES[dtype])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dt, M, K, N, zeros = (case[k] for k in ("kind", "dtype", "M", "K", "N", "zeros"))
    dev = torch.device("cuda", torch.cuda.current_device())
    s = {"kind": kind, "case": case}
    if kind in ("linear", "host"):
        s["w"] = PackedWeight.from_dense(_ternary(gen, K, N, zeros), scale=SCALE, device=dev)
        if kind == "linear":
            s["x"] = _activations(gen, (M, K), dt)
        else:
            s["x"] = _activations(gen, (K, M) if case["col_major"] else (M, K), dt).cpu().numpy()
    elif kind == "lists":
        w = _ternary(gen, K, N, zeros).astype(np.int32)
        tile = ter_spmm.tile_size_for(K)
        idx, off, til = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), tile, False, 4, as_numpy=True)
        s["lists"] = (torch.from_numpy(idx).to(torch.int16).to(dev), torch.from_numpy(off).to(dev), torch.from_numpy(til).to(torch.int16).to(dev))
        s["x"] = _activations(gen, (1, M, K), dt)
    elif kind == "mlp":
        s["mlp"] = PackedMLP(_ternary(gen, K, N, zeros), _ternary(gen, K, N, zeros), _ternary(gen, N, K, zeros), 0.0371, 0.0293, SCALE, device=dev)
        s["x"] = _activations(gen, (M, K), dt)
    elif kind == "module":
        cfg = TernaryConfig(hidden_size=K, intermediate_size=N, sparsity=zeros)
        s["module"] = LlamaTernaryMLP(cfg, scales=(0.0371, 0.0293, SCALE), generator=torch.Generator().manual_seed(seed))
        s["module"].packed(dev)
        s["x"] = _activations(gen, (1, M, K), dt)
    elif kind == "attn":
        cfg = TernaryConfig(hidden_size=K, num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], sparsity=zeros)
        s["module"] = LlamaTernaryAttention(cfg, scales=(SCALE,) * 4, generator=torch.Generator().manual_seed(seed))
        s["module"].packed_qkv(dev)
        s["module"].o_proj.packed(dev)
        s["x"] = _activations(gen, (1, M, K), dt)
    else:
        s["layer"] = layer = TernaryDecoderLayerTP(K, N, case["heads"], case["kv_heads"], K // case["heads"], zeros, 1, 0, dev, dtype=DTYPES[dt],
                                                   kv_len=KV_LEN, max_batch=M, seed=seed % 100003)
        s["x0"] = _activations(gen, (M, K), dt)
        s["x"] = torch.empty_like(s["x0"])

        def step():
            s["x"].copy_(s["x0"])
            x, pending = layer(s["x"])
            return layer.finish(x, pending)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side), torch.no_grad():
            step()
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]), torch.no_grad():
            s["y"] = step()
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["w"].matmul(s["x"])
    if kind == "host":
        col = s["case"]["col_major"]
        return s["w"].matmul_host(s["x"], col_major=col, y_col_major=col)
    if kind == "lists":
        c = s["case"]
        idx, off, til = s["lists"]
        return ter_spmm.ter_spmm(s["x"], idx, off, til, 1, c["M"], c["N"], c["K"], False, False, SCALE)
    if kind == "mlp":
        return s["mlp"].forward(s["x"])
    if kind == "layer":
        s["graph"].replay()
        return s["y"]
    with torch.no_grad():
        y = s["module"](s["x"])
    return y if kind == "module" else y[0]


def work(case):
    """Each weight read once at two bits per entry (the index arrays as they are for `lists`), activations in, results
    out; operations as a dense product counts them, which is how the tensor cores do it."""
    kind, M, K, N, e = case["kind"], case["M"], case["K"], case["N"], BYTES[case["dtype"]]
    if kind in ("linear", "host"):
        return {"bytes": K * N / 4 + M * K * e + M * N * (4 if case["dtype"] == "i8" else e), "flops": 2.0 * M * K * N}
    if kind == "lists":
        lists = 2 * K * N * (1 - case["zeros"]) + 16 * N * -(-K // ter_spmm.tile_size_for(K))
        return {"bytes": lists + M * (K + N) * e, "flops": 2.0 * M * K * N}
    if kind in ("mlp", "module"):
        return {"bytes": 3 * K * N / 4 + 2 * M * K * e, "flops": 6.0 * M * K * N}
    hd = K // case["heads"]
    proj = K * (K + 2 * case["kv_heads"] * hd) + K * K          # q | k | v and o
    if kind == "attn":
        return {"bytes": proj / 4 + 2 * M * K * e, "flops": 2.0 * M * proj + 2.0 * M * M * K}
    return {"bytes": (proj + 3 * K * N) / 4 + 2 * M * K * e + 2 * M * case["kv_heads"] * KV_LEN * hd * e,
            "flops": 2.0 * M * (proj + 3 * K * N) + 4.0 * M * KV_LEN * K}


def tolerance(case):
    if case["dtype"] == "i8":
        return "exact"
    one = {"f32": 1e-5, "f16": 1e-3, "bf16": 5e-3}[case["dtype"]]       # sums in fp32, one rounding of the result
    several = {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]   # intermediate results in the same type
    return {"rel": one if case["kind"] in ("linear", "host", "lists") else several}
