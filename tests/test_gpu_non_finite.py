"""Inf, NaN and activations near the end of the fp32 range through the two kernels on bit tiles and the calls that use them.

An activation touches the columns whose weight there is not zero, as in the product on index lists: Inf gives +-Inf there, NaN gives
NaN, and every other column is as if it were not there.  Only a product of many rows of 16-bit activations that are read in place
multiplies the zeros too (0 * Inf = NaN).  The reference is the same sum in fp64; finite sums are held to the bounds of the other tests,
1e-5 of the row's largest finite output."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, PackedWeight, _lib, ter_spmm

pytestmark = pytest.mark.gpu
DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
INF, NAN = float("inf"), float("nan")


def special_rows(X, big):
    """Rows 0 .. 3 (as many as there are) get what the test is about; the others stay as they are."""
    for row, at in ((0, {5: INF}), (1, {700: NAN}), (2, {5: INF, 6: -INF}), (3, {7: big, 8: big, 9: -big})):
        if row < X.shape[0]:
            for k, v in at.items():
                X[row, k] = v
    return X


def product(X, w, dense=False):
    """fp64, zeros of w left out (or not)."""
    X, w = X.double(), torch.as_tensor(w, device=X.device).double()
    Y = torch.where(torch.isfinite(X), X, 0.0) @ w
    for m in torch.nonzero(~torch.isfinite(X).all(1)).flatten().tolist():
        p = X[m, :, None] * w
        Y[m] = (p if dense else torch.where(w == 0, 0.0, p)).sum(0)
    return Y


def check(got, want, tol):
    got = got.double()
    want = torch.where(want.abs() > torch.finfo(torch.float32).max, want * INF, want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)]) and torch.equal(torch.isinf(got), torch.isinf(want))
    for g, r in zip(got, want):
        ok = torch.isfinite(r)
        assert not ok.any() or float((g[ok] - r[ok]).abs().max()) <= tol * float(r[ok].abs().max())


def weights(K, N, s, seed):
    w = random_ternary(np.random.default_rng(seed), K, N, s)
    w[5:10, :] = 0
    w[5, :N // 4], w[6, N // 8:N // 2] = 1, -1                 # Inf alone, both, -Inf alone
    w[7, N // 2:], w[8, N - 20:], w[9, N - 10:] = 1, 1, 1      # big alone, twice (past the range of fp32), two and one back
    return w


# one row and a few (decoded in registers), 24 and 200 (batched, with a hand-over between blocks and without); odd slices, ragged columns
@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("M", [1, 8, 24, 200])
@pytest.mark.parametrize("K,N", [(1000, 300), (4096, 1536)])
def test_product(K, N, M, dtype):
    w = weights(K, N, 0.6, K)
    pw = PackedWeight.from_dense(w)
    big = 4.0e4 if dtype == "f16" else 2.5e38
    X = special_rows(torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).to(DT[dtype]), big)
    out = torch.empty((M, N), device="cuda")
    L = _lib.lib()
    b0 = L.tllm_bits_launch_count()
    pw.matmul(X, out=out)
    decoded = L.tllm_bits_launch_count() > b0
    assert decoded or M > 1
    check(out, product(X, w, dense=dtype != "f32" and not decoded), 1e-5)
    pw.matmul(X.t().contiguous(), out=out, col_major=True)     # through planes where it is batched
    check(out, product(X, w), 1e-5)
    pw.check()
    pw.close()


# pairs of blocks, whole tiles and ranges of units, read in place (the zeros count) and through planes
@pytest.mark.parametrize("M,K,N,dtype,cut,dense", [(2177, 792, 1635, "bf16", 0, True), (2177, 792, 1635, "f16", 0, True), (2127, 778, 1854, "bf16", 0, False),
                                                   (880, 1085, 138, "f32", 0, False), (232, 6512, 2337, "f32", 1, False)])
def test_pairs_of_blocks(M, K, N, dtype, cut, dense):
    w = weights(K, N, 0.6, K)
    pw = PackedWeight.from_dense(w)
    X = special_rows(torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)).to(DT[dtype]), 4.0e4 if dtype == "f16" else 2.5e38)
    out = torch.empty((M, N), device="cuda")
    pw.matmul(X, out=out)
    plan = (ctypes.c_int * 5)()
    assert _lib.lib().tllm_mma_last_plan(plan) == 0 and tuple(plan)[:3] == (2, 2, cut), tuple(plan)
    check(out, product(X, w, dense=dense), 1e-5)
    pw.check()
    pw.close()


@pytest.mark.parametrize("dtype", list(DT))
def test_lists(dtype):
    K, N, T, M = 2048, 512, 256, 40                            # enough to be turned into bit tiles
    w = weights(K, N, 0.6, 3).astype(np.int32)
    idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), T, False, 4, as_numpy=True)
    ri, co = torch.tensor(idx.astype(np.int16), device="cuda"), torch.tensor(off.astype(np.int32), device="cuda")
    for m in (24, M):
        X = torch.randn((1, m, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).to(DT[dtype])
        special_rows(X[0], 4.0e4 if dtype == "f16" else 1.0e38)
        eps = {"f32": 0.0, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]
        want = product(X[0], w)
        if dtype == "f16":
            want = torch.where(want.abs() >= 65520, want * INF, want)              # what rounds to Inf in fp16
        check(ter_spmm.ter_spmm(X, ri, co, None, 1, m, N, K, False, False, tile_k=T)[0], want, 1e-5 + eps)


@pytest.mark.parametrize("M", [4, 200])
def test_fused_mlp(M):
    hidden, inter = 1024, 1536
    wg, wu, wd = weights(hidden, inter, 0.97, 1), weights(hidden, inter, 0.97, 2), random_ternary(np.random.default_rng(3), inter, hidden, 0.998)
    mlp = PackedMLP(wg, wu, wd, 0.05, 0.04, 0.03)
    X = special_rows(torch.randn((M, hidden), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M)), 100.0)
    g, u = product(X, wg) * 0.05, product(X, wu) * 0.04
    want = product((g * u / (1 + torch.exp(-g))).float(), wd) * 0.03
    assert torch.isfinite(want[:3]).any(1).all() and not torch.isfinite(want[:3]).all(1).any()
    check(mlp.forward(X), want, 1e-5 + 2.0 ** -22)
    mlp.close()


# Four columns a thread add up the warps' sums (more than thirty-two of them a block): the ones beside a sum that is not finite keep every bit
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_neighbours_of_a_sum_that_is_not_finite(dtype):
    M, K = 8, 1000
    N = 16 * 5 * torch.cuda.get_device_properties(0).multi_processor_count - 6
    w = random_ternary(np.random.default_rng(1), K, N, 0.5)
    w[7] = 0
    w[7, 1::5] = 1                                             # 2 * 2.5e38 is past the range of fp32 inside the kernel
    pw = PackedWeight.from_dense(w)
    X = torch.randn((M, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).to(DT[dtype])
    X[:, 7] = 0
    L = _lib.lib()
    b0 = L.tllm_bits_launch_count()
    plain = pw.matmul(X, out=torch.empty((M, N), device="cuda"))
    X[:, 7] = 2.5e38
    got = pw.matmul(X, out=torch.empty((M, N), device="cuda"))
    assert L.tllm_bits_launch_count() == b0 + 2
    used = torch.zeros(N, dtype=torch.bool)
    used[1::5] = True
    assert torch.equal(got[:, ~used], plain[:, ~used])
    check(got, product(X, w), 1e-5)
    pw.close()


# the same for pairs of gate and up columns: h comes back through a second product that takes one entry a column
def test_neighbours_of_a_gate_that_is_not_finite():
    M, hidden, inter = 8, 1000, 34 * torch.cuda.get_device_properties(0).multi_processor_count + 6
    wg, wu = random_ternary(np.random.default_rng(1), hidden, inter, 0.5), random_ternary(np.random.default_rng(2), hidden, inter, 0.5)
    wg[7], wu[7] = 0, 0
    wg[7, 1::5] = 1
    mlp = PackedMLP(wg, wu, np.eye(inter, hidden, dtype=np.int8), 0.05, 0.04, 1.0)
    X = torch.randn((M, hidden), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    X[:, 7] = 0
    L = _lib.lib()
    b0 = L.tllm_bits_launch_count()
    plain = mlp.forward(X).clone()
    X[:, 7] = 2.5e38
    got = mlp.forward(X)
    assert L.tllm_bits_launch_count() >= b0 + 2
    used = torch.zeros(hidden, dtype=torch.bool)
    used[1::5] = True
    assert torch.equal(got[:, ~used], plain[:, ~used]) and not torch.equal(got[:, used], plain[:, used])
    mlp.close()
