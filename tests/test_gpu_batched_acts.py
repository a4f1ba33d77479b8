"""The batched tensor-core product on every form of activations (csrc/mma_kernel.cuh): fp32 as three bf16 planes, int8 as fp16,
column-major and unaligned rows, at row counts around the edges of its row tiles; tiles that many blocks share.

Exact on integers (sums below 2^24); on N(0,1) within 1e-5 of the largest output, the bound of the other tensor-core kernels
(fp32 sums of exact products).
"""
import numpy as np
import pytest
import torch

import oracle
from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, PackedWeight, _lib

pytestmark = pytest.mark.gpu
DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i8": torch.int8}


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("K,N,s", [(40, 17, 0.3), (64, 130, 0.5), (1003, 517, 0.6), (4100, 128, 0.5)])
def test_exact_on_integer_activations(K, N, s, dtype):
    rng = np.random.default_rng(K + N)
    w = random_ternary(rng, K, N, s)
    pw = PackedWeight.from_dense(w)
    top = {"f32": 512, "f16": 512, "bf16": 127, "i8": 127}[dtype]
    for M in (129, 257, 300, 1200):
        xs = rng.integers(-top, top + 1, size=(M, K)).astype(np.float64)
        X = torch.tensor(xs, dtype=DT[dtype], device="cuda")
        out = torch.full((M, N), -1, dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
        want = oracle.dense_f64(xs, w)
        assert np.array_equal(pw.matmul(X, out=out).double().cpu().numpy(), want), M
        out.fill_(-1)
        assert np.array_equal(pw.matmul(X.t().contiguous(), out=out, col_major=True).double().cpu().numpy(), want), M
    pw.check()
    pw.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
def test_gaussian_activations(dtype):
    rng = np.random.default_rng(5)
    K, N = 4096, 2816
    w = random_ternary(rng, K, N, 0.6)
    pw = PackedWeight.from_dense(w, scale=0.03125)
    for M in (20, 64, 200, 512):
        X = torch.tensor(rng.standard_normal((M, K)), dtype=DT[dtype], device="cuda")
        ref = oracle.dense_f64(X.double().cpu().numpy(), w, 0.03125)
        Y = pw.matmul(X, out=torch.empty((M, N), dtype=torch.float32, device="cuda"))
        assert np.max(np.abs(Y.double().cpu().numpy() - ref)) <= 1e-5 * np.max(np.abs(ref)), M
    pw.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("hidden,inter", [(520, 1416), (768, 1027)])
def test_fused_mlp(dtype, hidden, inter):
    rng = np.random.default_rng(6)
    wg, wu, wd = (random_ternary(rng, *shape, 0.6) for shape in ((hidden, inter), (hidden, inter), (inter, hidden)))
    mlp = PackedMLP(wg, wu, wd, 0.021, 0.034, 0.027)
    for M in (40, 130, 300):
        X = torch.tensor(rng.standard_normal((M, hidden)), dtype=DT[dtype], device="cuda")
        ref = oracle.mlp_f64(X.double().cpu().numpy(), wg, wu, wd, 0.021, 0.034, 0.027, h_round={"f32": 3, "f16": 1, "bf16": 2}[dtype])
        err = np.max(np.abs(mlp.forward(X).double().cpu().numpy() - ref)) / np.max(np.abs(ref))
        # fp32 sums, and up to one last place of the type in h and in the result
        assert err <= 1e-5 + {"f32": 2.0 ** -22, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}[dtype], (M, err)
    mlp.close()


def test_calls_with_a_workspace_replay_from_a_graph():
    rng = np.random.default_rng(7)
    K, N, M = 1024, 640, 200
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    X = torch.zeros((M, K), device="cuda")
    pw.matmul(X)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        Y = pw.matmul(X)
        Z = pw.matmul(X * 2)
    for seed in range(3):
        xs = np.random.default_rng(seed).integers(-9, 10, size=(M, K)).astype(np.float64)
        X.copy_(torch.tensor(xs, dtype=torch.float32))
        g.replay()
        want = oracle.dense_f64(xs, w)
        assert np.array_equal(Y.double().cpu().numpy(), want) and np.array_equal(Z.double().cpu().numpy(), 2 * want)
    pw.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("K,N", [(512, 256), (1000, 130), (2048, 2048), (4352, 257), (2100, 3900), (1024, 9000), (7000, 128)])
def test_few_tiles(K, N, dtype):
    """Products of few tiles, which clusters of two, four and eight blocks share: exact on integers, row- and column-major, at
    row counts around the sixteens that a cluster divides among its blocks."""
    g = torch.Generator(device="cuda").manual_seed(K + N)
    w = torch.randint(-1, 2, (K, N), generator=g, device="cuda", dtype=torch.int8)
    pw = PackedWeight.from_dense(w.cpu().numpy())
    prev = _lib.lib().tllm_set_mma_min_rows(1 if dtype != "f32" else -1)
    try:
        for M in (1, 16, 17, 33, 48, 64, 80, 128, 131, 200, 256):
            X = torch.randint(-16, 17, (M, K), generator=g, device="cuda").to(DT[dtype])
            want = X.double() @ w.double()
            out = torch.full((M, N), -1, dtype=torch.float32, device="cuda")
            assert torch.equal(pw.matmul(X, out=out).double(), want), M
            out.fill_(-1)
            assert torch.equal(pw.matmul(X, out=out).double(), want), M
            assert float((pw.matmul(X).double() - want).abs().max()) <= {"f32": 0.0, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype] * float(want.abs().max())
        pw.check()
    finally:
        _lib.lib().tllm_set_mma_min_rows(prev)
    pw.close()
