"""The register-decode product (two-bit tiles of W decoded into mma.sync fragments, csrc/bits_kernel.cuh) against the
oracle, through the calls that reach it by default: few activation rows of any type and layout.

Integer-valued activations are exact (products and partial sums are integers below 2^24); on N(0,1) the fp32 sums of
exact products stay within 1e-5 of the largest output, the bound the other tensor-core kernels are held to.
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, PackedWeight, _lib

pytestmark = pytest.mark.gpu
DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i8": torch.int8}


def decoded(call, *args, **kw):
    """The result of a call, which has to have run on the register decoder and nothing else."""
    L = _lib.lib()
    b0, n0 = L.tllm_bits_launch_count(), L.tllm_launch_count()
    y = call(*args, **kw)
    assert L.tllm_bits_launch_count() - b0 == L.tllm_launch_count() - n0 > 0
    return y


def bits_plan():
    plan = (ctypes.c_int * 6)()
    assert _lib.lib().tllm_bits_last_plan(plan) == 0
    return tuple(plan)


# one slice, an odd last slice, K and N multiples of nothing (rows of X on odd addresses), fewer pairs of slices than
# warps, several passes per block (more than eight groups of sixteen columns per SM)
SHAPES = [(1, 1, 0.0), (40, 17, 0.3), (64, 16, 0.5), (77, 5, 0.3), (192, 48, 0.5), (1003, 517, 0.6), (1000, 70, 0.6), (2056, 386, 0.9), (4099, 33, 0.5), (520, 21000, 0.5)]


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("K,N,s", SHAPES)
def test_exact_on_integer_activations(K, N, s, dtype):
    rng = np.random.default_rng(K + N)
    w = random_ternary(rng, K, N, s)
    pw = PackedWeight.from_dense(w)
    top = {"f32": 512, "f16": 512, "bf16": 127, "i8": 127}[dtype]
    for M in (1, 2, 3, 7, 8, 9, 16, 17, 32):
        # with more rows, of fp32 and column-major ones sooner, the choice depends on the shape
        any_kernel = lambda call, *args, **kw: call(*args, **kw)
        run = decoded if M <= 3 or M <= 8 and dtype != "f32" else any_kernel
        run_columns = decoded if M == 1 or M <= 3 and N != 21000 else any_kernel
        run_offset = run_columns if dtype == "f32" and N == 21000 else run
        xs = rng.integers(-top, top + 1, size=(M, K)).astype(np.float64)
        X = torch.tensor(xs, dtype=DT[dtype], device="cuda")
        out = torch.full((M, N), -1, dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
        want = oracle.dense_f64(xs, w)
        assert np.array_equal(run(pw.matmul, X, out=out).double().cpu().numpy(), want), M
        out.fill_(-1)
        assert np.array_equal(run_columns(pw.matmul, X.t().contiguous(), out=out, col_major=True).double().cpu().numpy(), want), M
        # rows that start inside a wider buffer, on an address that is a multiple of the element size only
        buf = torch.zeros(M * K + 1, dtype=DT[dtype], device="cuda")
        buf[1:] = X.reshape(-1)
        assert np.array_equal(run_offset(pw.matmul, buf[1:].view(M, K), out=out).double().cpu().numpy(), want), M
    pw.check()
    pw.close()


# int8 sums are int32: the largest values of one sign, at the row counts around the blocks of eight, sixteen and thirty-two rows
@pytest.mark.parametrize("M", [8, 9, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("K,N", [(64, 16), (130, 517), (8200, 40)])
def test_int8_extremes(K, N, M):
    w = random_ternary(np.random.default_rng(M), K, N, 0.3)
    w[:, 0], w[:, 1] = 1, -1
    pw = PackedWeight.from_dense(w)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(K))
    x[0], x[-1] = -128, 127
    want = x.double() @ torch.tensor(w, device="cuda").double()
    assert torch.equal(pw.matmul(x).double(), want)
    assert torch.equal(pw.matmul(x.t().contiguous(), col_major=True).double(), want)
    pw.close()


# Activations that all warps of a block share: columns cut two and four ways and several passes (groups of sixteen columns per SM), X in one chunk and in two
# (16 and 17, 32 and 33 pairs of slices), ends of K inside a slice, fewer pairs than warps; rows on 16 bytes, on odd addresses and columns.
@pytest.mark.parametrize("groups", [3, 5, 7, 13])
@pytest.mark.parametrize("dtype,M,K", [("f16", 1, 4104), ("f16", 8, 4096), ("bf16", 8, 4232), ("bf16", 16, 2048), ("f16", 16, 2184), ("f32", 6, 2048), ("f32", 7, 2180),
                                       ("f32", 8, 4228), ("f32", 1, 4100), ("i8", 1, 4112), ("i8", 9, 2192), ("i8", 32, 4096), ("i8", 17, 1168), ("f16", 8, 1000)])
def test_shared_activations(dtype, M, K, groups):
    rng = np.random.default_rng(K + groups)
    N = 16 * groups * torch.cuda.get_device_properties(0).multi_processor_count - 5
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=torch.Generator().manual_seed(K))
    pw = PackedWeight.from_dense(w.numpy())
    top = 127 if dtype in ("i8", "bf16") else 512
    X = torch.tensor(rng.integers(-top, top + 1, size=(M, K)), dtype=DT[dtype], device="cuda")
    want = X.double() @ w.cuda().double()
    out = torch.empty((M, N), dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
    buf = torch.zeros(M * K + 1, dtype=DT[dtype], device="cuda")
    buf[1:] = X.reshape(-1)
    for x, kw in ((X, {}), (buf[1:].view(M, K), {}), (X.t().contiguous(), {"col_major": True})):
        out.fill_(-1)
        assert torch.equal(pw.matmul(x, out=out, **kw).double(), want)
    pw.check()
    pw.close()


# Shared activations take the room of what they hold, not of chunks rounded up to sixteen pairs of slices: K just above 4096 and 2048, up to the last row that fits
@pytest.mark.parametrize("dtype,M,K,N", [("f16", 12, 5120, 5120), ("bf16", 13, 5120, 10240), ("bf16", 14, 5120, 5120), ("bf16", 16, 4224, 11008), ("f32", 6, 5120, 5120), ("f32", 8, 2304, 8192),
                                         ("i8", 32, 4224, 8192), ("i8", 32, 5120, 5120)])
def test_shared_activations_as_they_fit(dtype, M, K, N):
    rng = np.random.default_rng(K)
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=torch.Generator().manual_seed(N))
    pw = PackedWeight.from_dense(w.numpy())
    top = 127 if dtype in ("i8", "bf16") else 512
    X = torch.tensor(rng.integers(-top, top + 1, size=(M, K)), dtype=DT[dtype], device="cuda")
    out = torch.empty((M, N), dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
    for _ in range(2):
        out.fill_(-1)
        assert torch.equal(decoded(pw.matmul, X, out=out).double(), X.double() @ w.cuda().double())
        assert bits_plan()[4] == 2
    pw.check()
    pw.close()


# Columns, and rows on odd addresses, that the warps share although no split fetches them twice: a K of one pair of slices to a warp, of fewer and of more of them,
# in one chunk and in two
@pytest.mark.parametrize("dtype,M,K,N,columns,chunks", [("i8", 9, 1344, 1152, True, 1), ("i8", 5, 900, 811, True, 1), ("i8", 2, 2188, 640, True, 1), ("bf16", 5, 1728, 2304, True, 1), ("f16", 3, 896, 811, True, 1),
                                                        ("f16", 4, 2376, 1043, True, 2), ("f32", 3, 720, 1024, True, 1), ("f32", 2, 1192, 384, True, 1), ("i8", 24, 1827, 1280, False, 1), ("i8", 1, 4104, 333, False, 1),
                                                        ("f16", 7, 2376, 2048, False, 2), ("bf16", 5, 768, 4864, False, 1), ("f16", 2, 1480, 640, False, 1), ("f32", 4, 516, 320, False, 1)])
def test_shared_without_a_split(dtype, M, K, N, columns, chunks):
    gen = torch.Generator().manual_seed(K)
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=gen)
    pw = PackedWeight.from_dense(w.numpy())
    X = torch.randint(-127, 128, (M, K), generator=gen).to(DT[dtype]).cuda()
    buf = torch.zeros(M * K + 1, dtype=DT[dtype], device="cuda")
    buf[1:] = X.reshape(-1)
    x = X.t().contiguous() if columns else buf[1:].view(M, K)
    out = torch.full((M, N), -1, dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
    assert torch.equal(decoded(pw.matmul, x, out=out, col_major=columns).double(), X.double() @ w.cuda().double())
    assert bits_plan()[2:5] == (1, 1, chunks)
    pw.check()
    pw.close()


# The forms of shared activations, each by the plan of its launch: columns cut two and four ways, one pass and more of them, X in one chunk and in two; rows on 16
# bytes, on odd addresses and columns
@pytest.mark.parametrize("access,dtype,M,K,groups,split,passes,chunks", [
    ("rows", "f16", 8, 4096, 5, 2, 1, 2), ("rows", "bf16", 8, 4232, 7, 4, 1, 2), ("rows", "bf16", 16, 2048, 5, 4, 1, 1), ("rows", "f16", 8, 4096, 13, 4, 2, 2), ("rows", "f32", 6, 2048, 5, 4, 1, 1),
    ("rows", "f32", 7, 2180, 5, 4, 1, 2), ("rows", "f32", 8, 1160, 3, 2, 1, 1), ("rows", "f32", 5, 520, 13, 4, 2, 1), ("rows", "i8", 32, 4096, 3, 4, 1, 2), ("rows", "i8", 32, 4096, 5, 4, 2, 2),
    ("rows", "i8", 17, 1168, 7, 4, 2, 1), ("rows", "i8", 9, 2192, 13, 4, 2, 2), ("rows", "f16", 1, 4104, 5, 2, 1, 1),
    ("offset", "f16", 8, 4096, 5, 2, 1, 2), ("offset", "f16", 8, 1000, 7, 4, 1, 1), ("offset", "f16", 4, 1003, 13, 4, 2, 1), ("offset", "bf16", 12, 1000, 5, 4, 1, 1), ("offset", "f32", 4, 1016, 3, 2, 1, 1),
    ("offset", "f32", 5, 520, 7, 4, 1, 1), ("offset", "i8", 8, 4100, 13, 4, 2, 2), ("offset", "i8", 17, 1168, 5, 4, 2, 1), ("offset", "i8", 16, 1040, 13, 4, 2, 1),
    ("columns", "f16", 4, 1003, 5, 2, 1, 1), ("columns", "f16", 8, 1000, 13, 4, 2, 1), ("columns", "bf16", 12, 1000, 7, 4, 1, 1), ("columns", "f16", 8, 4096, 13, 4, 2, 2), ("columns", "f32", 5, 520, 5, 4, 1, 1),
    ("columns", "f32", 4, 1016, 7, 4, 1, 1), ("columns", "f32", 2, 4100, 5, 2, 1, 2), ("columns", "i8", 8, 4100, 13, 4, 2, 2)])
def test_forms_of_shared_activations(access, dtype, M, K, groups, split, passes, chunks):
    gen = torch.Generator().manual_seed(K + groups)
    N = 16 * groups * torch.cuda.get_device_properties(0).multi_processor_count - 5
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=gen)
    pw = PackedWeight.from_dense(w.numpy())
    top = 127 if dtype in ("i8", "bf16") else 512
    X = torch.randint(-top, top + 1, (M, K), generator=gen).to(DT[dtype]).cuda()
    buf = torch.zeros(M * K + 1, dtype=DT[dtype], device="cuda")
    buf[1:] = X.reshape(-1)
    x = {"rows": X, "offset": buf[1:].view(M, K), "columns": X.t().contiguous()}[access]
    want = X.double() @ w.cuda().double()
    out = torch.empty((M, N), dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
    for _ in range(2):
        out.fill_(-1)
        assert torch.equal(decoded(pw.matmul, x, out=out, col_major=access == "columns").double(), want)
        assert bits_plan()[2:5] == (split, passes, chunks)
    pw.check()
    pw.close()


# Four columns per thread with results of 16 bits, stored together and one by one, one of the four not finite and none
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("M,groups", [(8, 5), (16, 3)])
def test_sums_of_the_warps_in_16_bits(dtype, M, groups):
    K, sms = 120, torch.cuda.get_device_properties(0).multi_processor_count      # sums of up to 120 are exact in both types
    gen = torch.Generator().manual_seed(M)
    for n in (16 * groups * sms, 16 * groups * sms - 4, 16 * groups * sms - 6):
        w = torch.randint(-1, 2, (K, n), dtype=torch.int8, generator=gen)
        w[0] = 0
        w[0, 5], w[0, n - 1] = 1, -1
        pw = PackedWeight.from_dense(w.numpy())
        X = torch.randint(-1, 2, (M, K), generator=gen).to(DT[dtype]).cuda()
        want = X.double() @ w.cuda().double()
        out = torch.full((M * n + 1,), -1, dtype=DT[dtype], device="cuda")
        for y in (out[:-1].view(M, n), out[1:].view(M, n)):
            assert torch.equal(decoded(pw.matmul, X, out=y).double(), want)
        X[M - 1, 0] = float("inf")
        want[M - 1, 5], want[M - 1, n - 1] = float("inf"), -float("inf")
        for y in (out[:-1].view(M, n), out[1:].view(M, n)):
            y.fill_(-1)
            assert torch.equal(decoded(pw.matmul, X, out=y).double(), want)
        pw.close()


# Gate and up columns that four-column threads add up: more than thirty-two (group, row) pairs a block
@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("M", [6, 8])
def test_wide_fused_mlp(dtype, M):
    rng = np.random.default_rng(M)
    hidden, inter = 264, 40 * torch.cuda.get_device_properties(0).multi_processor_count + 2
    wg, wu, wd = (random_ternary(rng, *shape, 0.6) for shape in ((hidden, inter), (hidden, inter), (inter, hidden)))
    mlp = PackedMLP(wg, wu, wd, 0.021, 0.034, 0.027)
    X = torch.tensor(rng.standard_normal((M, hidden)), dtype=DT[dtype], device="cuda")
    ref = oracle.mlp_f64(X.double().cpu().numpy(), wg, wu, wd, 0.021, 0.034, 0.027, h_round={"f32": 3, "f16": 1, "bf16": 2}[dtype])
    L = _lib.lib()
    b0 = L.tllm_bits_launch_count()
    got = mlp.forward(X)
    assert L.tllm_bits_launch_count() > b0
    err = np.max(np.abs(got.double().cpu().numpy() - ref)) / np.max(np.abs(ref))
    assert err <= 1e-5 + {"f32": 2.0 ** -22, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}[dtype], err          # as in test_fused_mlp
    mlp.close()


# Results added up a column per thread and four per thread, stored together and one by one: around thirty-two (group, row) pairs per block, N a multiple of four and
# not, Y on 16 bytes and not, sums that are not finite among the four
@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("M,groups", [(8, 3), (8, 4), (8, 5), (1, 9), (16, 2), (16, 3), (32, 1), (32, 2)])
def test_sums_of_the_warps(dtype, M, groups):
    K, N = 520, 16 * groups * torch.cuda.get_device_properties(0).multi_processor_count
    gen = torch.Generator().manual_seed(M)
    for n in (N, N - 4, N - 6):
        w = torch.randint(-1, 2, (K, n), dtype=torch.int8, generator=gen)
        w[0] = 0
        w[0, 5], w[0, n - 1] = 1, -1
        pw = PackedWeight.from_dense(w.numpy())
        X = torch.randint(-64, 65, (M, K), generator=gen).to(DT[dtype]).cuda()
        want = X.double() @ w.cuda().double()
        out = torch.full((M * n + 1,), -1, dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
        for y in (out[:-1].view(M, n), out[1:].view(M, n)):
            assert torch.equal(pw.matmul(X, out=y).double(), want)
        if dtype != "i8":
            X[M - 1, 0] = float("inf")
            want[M - 1, 5], want[M - 1, n - 1] = float("inf"), -float("inf")
            got = pw.matmul(X, out=out[:-1].view(M, n)).double()
            same = want.clone()
            if not torch.equal(got, same):                           # many rows of 16-bit activations multiply the zeros too: 0 * Inf
                assert dtype != "f32" and M > 8 and torch.equal(torch.isnan(got[M - 1]), ~torch.isinf(want[M - 1])) and torch.equal(got[:-1], want[:-1])
        pw.close()


# Four blocks of columns of B in registers, rows on 16 bytes: several pairs of slices per warp, slots that are used again, the columns cut two and
# four ways.
@pytest.mark.parametrize("M", [17, 24, 31, 32])
@pytest.mark.parametrize("K,N", [(2048, 8192), (4096, 4096)])
def test_int8_of_32_rows_in_registers(K, N, M):
    w = random_ternary(np.random.default_rng(M), K, N, 0.3)
    w[:, 0], w[:, N - 1] = 1, -1
    pw = PackedWeight.from_dense(w)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(K))
    x[0], x[-1] = -128, 127
    assert torch.equal(decoded(pw.matmul, x).double(), x.double() @ torch.tensor(w, device="cuda").double())
    pw.close()


# the largest K that int8 takes here: sums of 2^24, accumulators of +-64 * 2^24
def test_int8_of_the_largest_k():
    K, N = 131072, 24
    w = random_ternary(np.random.default_rng(0), K, N, 0.3)
    w[:, 0], w[:, N - 1] = 1, -1
    pw = PackedWeight.from_dense(w)
    for value in (-128, 127):
        x = torch.full((1, K), value, dtype=torch.int8, device="cuda")
        assert torch.equal(decoded(pw.matmul, x).double(), x.double() @ torch.tensor(w, device="cuda").double())
        x = x.expand(8, K).contiguous()
        assert torch.equal(pw.matmul(x).double(), x.double() @ torch.tensor(w, device="cuda").double())
    pw.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
def test_gaussian_activations_and_result_types(dtype):
    rng = np.random.default_rng(5)
    K, N, s = 4096, 2816, 0.6
    w = random_ternary(rng, K, N, s)
    pw = PackedWeight.from_dense(w, scale=0.03125)
    for M in (1, 5, 16, 32):
        X = torch.tensor(rng.standard_normal((M, K)), dtype=DT[dtype], device="cuda")
        ref = oracle.dense_f64(X.double().cpu().numpy(), w, 0.03125)
        out = torch.empty((M, N), dtype=torch.float32, device="cuda")
        Y = decoded(pw.matmul, X, out=out) if M <= 8 else pw.matmul(X, out=out)
        assert np.max(np.abs(Y.double().cpu().numpy() - ref)) <= 1e-5 * np.max(np.abs(ref))
        eps = {"f32": 2.0 ** -23, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]          # one rounding to the result's type
        assert np.max(np.abs(pw.matmul(X).double().cpu().numpy() - ref)) <= (1e-5 + eps) * np.max(np.abs(ref))
    pw.close()


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
def test_fused_mlp(dtype):
    rng = np.random.default_rng(6)
    hidden, inter = 520, 1416
    wg, wu, wd = (random_ternary(rng, *shape, 0.6) for shape in ((hidden, inter), (hidden, inter), (inter, hidden)))
    mlp = PackedMLP(wg, wu, wd, 0.021, 0.034, 0.027)
    for M in (1, 8, 13):
        X = torch.tensor(rng.standard_normal((M, hidden)), dtype=DT[dtype], device="cuda")
        ref = oracle.mlp_f64(X.double().cpu().numpy(), wg, wu, wd, 0.021, 0.034, 0.027, h_round={"f32": 3, "f16": 1, "bf16": 2}[dtype])
        err = np.max(np.abs(mlp.forward(X).double().cpu().numpy() - ref)) / np.max(np.abs(ref))
        # fp32 sums, and up to one last place of the type in h and in the result
        assert err <= 1e-5 + {"f32": 2.0 ** -22, "f16": 2.0 ** -10, "bf16": 2.0 ** -7}[dtype], (M, err)
    mlp.close()
