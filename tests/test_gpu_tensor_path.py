"""The tensor-core (tcgen05) product against the oracle, through the C ABI.

From a configurable number of activation rows on, fp16 / bf16 products run on the dense two-bit copy of W with
tcgen05.mma instead of the gather kernel.  The reference has no counterpart (its kernels gather for every M,
ternaryLLM_GPU/csrc/ter_spmm_kernel.cuh:106-308), so the pin is the oracle's dense fp64 product: bit-exact on
integer-valued activations (every product and every partial sum is an integer below 2^24, so the order of the
sums cannot matter), and within 1e-3 of the largest output on N(0,1) activations.
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, PackedWeight, _lib

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}
TOL = 1e-3


def dev():
    return torch.device("cuda", 0)


@pytest.fixture(autouse=True)
def tensor_kernel_from_eight_rows():
    """A fixed crossover, so that which kernel runs does not depend on the cost model (tested on its own below)."""
    L = _lib.lib()
    prev = L.tllm_set_mma_min_rows(8)
    yield
    L.tllm_set_mma_min_rows(prev)


def mma_launches():
    return _lib.lib().tllm_mma_launch_count()


SHAPES = [(64, 128, 0.5), (128, 256, 0.5), (1000, 70, 0.6), (4096, 1024, 0.75), (2056, 386, 0.5), (8192, 512, 0.9), (512, 4096, 0.5)]
ROWS = [8, 16, 17, 33, 64, 65, 130, 256, 300, 700]


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("K,N,s", SHAPES)
def test_exact_on_integer_activations(K, N, s, dtype):
    rng = np.random.default_rng(K + N)
    w = random_ternary(rng, K, N, s)
    pw = PackedWeight.from_dense(w, scale=1.0)
    assert pw.info["bit_tile_bytes"] == ((N + 127) // 128) * ((K + 63) // 64) * 2048
    for M in (ROWS if K * N <= 2 ** 20 else (8, 40, 129, 300)):
        xs = rng.integers(-4, 5, size=(M, K)).astype(np.float64)
        X = torch.tensor(xs, dtype=DT[dtype], device=dev())
        Y = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev())
        n0 = mma_launches()
        pw.matmul(X, out=Y)
        assert mma_launches() == n0 + 1, "the call did not run on the tensor-core kernel"
        want = oracle.dense_f64(xs, w, 1.0)
        assert np.array_equal(Y.double().cpu().numpy(), want), (K, N, M)
    pw.check()
    pw.close()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_tolerance_on_gaussian_activations_and_agreement_with_the_gather_kernel(dtype):
    rng = np.random.default_rng(11)
    K, N = 4096, 2816
    w = random_ternary(rng, K, N, 0.6)
    s = float(np.float16(0.0371))
    pw = PackedWeight.from_dense(w, scale=s)
    L = _lib.lib()
    for M in (8, 16, 48, 100, 512):
        X = torch.tensor(rng.standard_normal((M, K)), dtype=DT[dtype], device=dev())
        ref = oracle.dense_f64(X.double().cpu().numpy(), w, s)
        n0 = mma_launches()
        Y = pw.matmul(X)
        assert mma_launches() == n0 + 1
        eps = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]
        err = np.max(np.abs(Y.double().cpu().numpy() - ref)) / np.max(np.abs(ref))
        assert err <= TOL + eps, (M, err)
        # the gather kernel on the same handle, same inputs: both are within rounding of the fp64 product
        L.tllm_set_mma_min_rows(0)
        Yg = pw.matmul(X)
        L.tllm_set_mma_min_rows(8)
        assert mma_launches() == n0 + 1
        assert np.max(np.abs(Yg.double().cpu().numpy() - Y.double().cpu().numpy())) / np.max(np.abs(ref)) <= 2 * eps + 1e-5
    pw.check()
    pw.close()


def mma_plan():
    """Of the calling thread's last launch: slices of a unit, blocks that share an MMA, cut (0 tiles, 1 ranges of units, 2 clusters), blocks of a
    cluster, rows of a tile."""
    plan = (ctypes.c_int * 5)()
    assert _lib.lib().tllm_mma_last_plan(plan) == 0
    return tuple(plan)


# The forms of the kernel with units of two slices: blocks that share an MMA, cut, blocks of a cluster, whether a tile has more than 128 columns of
# D (two places in the ring of expanded units, else four).  Even and odd numbers of column tiles (of the last one a pair's second block has
# none), one slice and many, odd ones, activations that TMA reads in place and that it does not (K not a multiple of eight, fp32), several legs of fp32.  The
# sizes keep their form on GPUs where 28 to 35 clusters of four blocks and 13 to 17 of eight fit (33 and 15 where they were chosen).
@pytest.mark.parametrize("M,K,N,dtype,blocks,cut,cluster,wide", [
    (160, 2424, 9902, "f16", 2, 0, 1, True), (2177, 792, 1635, "bf16", 2, 0, 1, True), (2127, 778, 1854, "f16", 2, 0, 1, True),
    (880, 1085, 138, "f32", 2, 0, 1, True), (799, 1009, 263, "f32", 2, 0, 1, True),
    (2178, 208, 8140, "bf16", 2, 1, 1, True), (1577, 312, 14154, "f16", 2, 1, 1, True), (2204, 65, 9729, "bf16", 2, 1, 1, True),
    (1801, 144, 8836, "f16", 2, 1, 1, False), (1905, 88, 13945, "bf16", 2, 1, 1, False),
    (500, 4100, 2500, "f32", 2, 1, 1, True), (232, 6512, 2337, "f32", 2, 1, 1, True),
    (342, 256, 200, "f16", 1, 0, 1, False), (1906, 64, 539, "bf16", 1, 0, 1, True), (591, 348, 1800, "f32", 1, 0, 1, True),
    (1862, 80, 6850, "f16", 1, 1, 1, False), (2191, 64, 6630, "bf16", 1, 1, 1, True), (800, 5910, 294, "f32", 1, 1, 1, True),
    (784, 1985, 411, "f32", 1, 2, 2, True), (2210, 3123, 144, "bf16", 1, 2, 4, True), (264, 4646, 206, "f32", 1, 2, 8, True)])
def test_exact_on_units_of_two_slices(M, K, N, dtype, blocks, cut, cluster, wide):
    rng = np.random.default_rng(M + K)
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w, scale=1.0)
    x = torch.tensor(rng.integers(-4, 5, size=(M, K)), dtype=torch.float64, device=dev())
    n0 = mma_launches()
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev())
    L = _lib.lib()
    L.tllm_set_mma_min_rows(-1)                       # the library's choice, fp32 as well
    for _ in range(2):                                # the second launch starts beside the first one
        pw.matmul(x.to({"f32": torch.float32, **DT}[dtype]), out=y)
    assert mma_launches() == n0 + 2, "the call did not run on the tensor-core kernel"
    plan = mma_plan()
    assert plan[:4] == (2, blocks, cut, cluster) and (plan[4] * (3 if dtype == "f32" else 1) > 128) == wide, plan
    assert torch.equal(y.double(), x @ torch.tensor(w, device=dev()).double())
    pw.check()
    pw.close()


# Clusters of two and four pairs of blocks: one plane and three, ragged K, rows and columns, int8, gate and up; launches one behind the other
@pytest.mark.parametrize("M,K,N,dtype,cluster", [(256, 8192, 2048, "f32", 2), (100, 4160, 4096, "f32", 2), (512, 8300, 1000, "f32", 2), (400, 8300, 500, "f32", 4),
                                                 (700, 12352, 2048, "f16", 2), (700, 12352, 2041, "i8", 2)])
def test_exact_on_clusters_of_pairs(M, K, N, dtype, cluster):
    gen = torch.Generator().manual_seed(K + N)
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=gen)
    pw = PackedWeight.from_dense(w.numpy(), scale=1.0)
    L = _lib.lib()
    L.tllm_set_mma_min_rows(-1)
    X = torch.randint(-4, 5, (M, K), generator=gen).to({"f32": torch.float32, "f16": torch.float16, "i8": torch.int8}[dtype]).cuda()
    want = X.double() @ w.cuda().double()
    out = torch.full((M, N), -1, dtype=torch.int32 if dtype == "i8" else torch.float32, device="cuda")
    for x, kw in ((X, {}), (X, {}), (X.t().contiguous(), {"col_major": True})):
        pw.matmul(x, out=out, **kw)
        plan = mma_plan()
        assert plan[1:3] != (2, 2) or plan[3] == cluster, plan
        if not kw:
            assert plan[:4] == (2, 2, 2, cluster), plan
        assert torch.equal(out.double(), want)
    pw.check()
    pw.close()


def test_repeated_calls_and_row_counts_share_the_split_scratch():
    """Back-to-back launches with different row counts on one handle (programmatic dependent launch lets the
    next kernel start before the previous one has drained): counters and partial sums must not leak."""
    rng = np.random.default_rng(12)
    K, N = 8192, 1024                      # 8 column tiles over all SMs: every tile is shared by many blocks
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    outs = []
    for rep in range(3):
        for M in (64, 8, 33, 16):
            xs = rng.integers(-3, 4, size=(M, K)).astype(np.float64)
            X = torch.tensor(xs, dtype=torch.bfloat16, device=dev())
            Y = torch.empty((M, N), dtype=torch.float32, device=dev())
            pw.matmul(X, out=Y)
            outs.append((xs, Y))
    torch.cuda.synchronize()
    for xs, Y in outs:
        assert np.array_equal(Y.double().cpu().numpy(), oracle.dense_f64(xs, w, 1.0))
    pw.check()
    pw.close()


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_fused_mlp_on_the_tensor_path(dtype):
    rng = np.random.default_rng(13)
    hidden, inter = 1024, 2752
    wg, wu = random_ternary(rng, hidden, inter, 0.6), random_ternary(rng, hidden, inter, 0.6)
    wd = random_ternary(rng, inter, hidden, 0.6)
    sg, su, sd = (float(np.float16(v)) for v in rng.uniform(0.01, 0.05, 3))
    mlp = PackedMLP(wg, wu, wd, sg, su, sd)
    mode = {"f16": 1, "bf16": 2}[dtype]
    for M in (8, 32, 200):
        X = torch.tensor(rng.standard_normal((M, hidden)), dtype=DT[dtype], device=dev())
        ref = oracle.mlp_f64(X.double().cpu().numpy(), wg, wu, wd, sg, su, sd, h_round=mode)
        n0 = mma_launches()
        Y = mlp.forward(X).double().cpu().numpy()
        assert mma_launches() == n0 + 2
        eps = {"f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype]
        err = np.max(np.abs(Y - ref)) / np.max(np.abs(ref))
        assert err <= TOL + 4 * eps, (M, err)
    mlp.close()


def test_crossover_setting_and_fallbacks():
    L = _lib.lib()
    rng = np.random.default_rng(14)
    K, N = 1024, 256
    w = random_ternary(rng, K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    X = torch.tensor(rng.integers(-4, 5, size=(32, K)).astype(np.float32), device=dev())
    n0 = mma_launches()
    pw.matmul(X)                                            # fp32 activations stay on the gather kernel
    pw.matmul(X.to(torch.float16)[:4].contiguous())         # below the crossover
    assert mma_launches() == n0
    prev = L.tllm_set_mma_min_rows(2)
    assert prev == 8
    pw.matmul(X.to(torch.float16)[:4].contiguous())
    assert mma_launches() == n0 + 1
    assert L.tllm_set_mma_min_rows(8) == 2
    narrow = PackedWeight.from_dense(random_ternary(rng, 40, 256, 0.5))     # fewer rows of W than one TMA box: gather kernel
    Xn = torch.tensor(rng.integers(-4, 5, size=(32, 40)).astype(np.float32), dtype=torch.float16, device=dev())
    L.tllm_set_mma_min_rows(2)
    narrow.matmul(Xn)
    L.tllm_set_mma_min_rows(8)
    assert mma_launches() == n0 + 1
    narrow.close()
    lean = PackedWeight.from_dense(w, no_bit_tiles=1)       # no dense copy: always the gather kernel
    assert lean.info["bit_tile_bytes"] == 0
    Y = lean.matmul(X.to(torch.float16))
    assert mma_launches() == n0 + 1
    assert np.array_equal(Y.double().cpu().numpy(), oracle.dense_f64(X.double().cpu().numpy(), w, 1.0))
    pw.close()
    lean.close()


def test_cost_model_dispatch():
    """Default setting, by the launches of each kernel: one row of a wide, 90 %-sparse weight goes to the gather kernel (its index
    lists are shorter than two bits an entry) and a few rows of any weight to the register decoder; many rows go to the
    batched tensor-core kernel; a few 16-bit rows of a weight so wide that the decoder makes several passes go to the kernel on
    four-bit planes."""
    L = _lib.lib()
    L.tllm_set_mma_min_rows(-1)
    rng = np.random.default_rng(15)

    def launches():
        return np.array([L.tllm_bits_launch_count(), L.tllm_mma_launch_count(), L.tllm_nibble_launch_count(), L.tllm_launch_count()])

    for K, N, s, want in ((4096, 2816, 0.5, {1: "bits", 2: "bits", 4: "bits", 8: "bits", 64: "mma", 300: "mma"}),
                          (4096, 2816, 0.9, {1: "bits", 4: "bits", 64: "mma", 300: "mma"}),
                          (4096, 11008, 0.95, {1: "gather", 4: "bits", 300: "mma"}),
                          (8192, 28672, 0.5, {1: "nibble", 300: "mma"})):
        w = random_ternary(rng, K, N, s)
        pw = PackedWeight.from_dense(w)
        Wd = torch.tensor(w, device=dev()).double()
        for M, kernel in want.items():
            X = torch.tensor(rng.integers(-4, 5, size=(M, K)).astype(np.float32), dtype=torch.bfloat16, device=dev())
            Y = torch.empty((M, N), dtype=torch.float32, device=dev())
            n0 = launches()
            pw.matmul(X, out=Y)
            n = launches() - n0
            assert n[3] == 1 and list(n[:3]) == [kernel == "bits", kernel == "mma", kernel == "nibble"], (K, N, s, M, kernel, n)
            assert torch.equal(Y.double(), X.double() @ Wd)
        pw.close()


# Default setting, activations that the register decoder cannot read by asynchronous copies, or (fp32, wide weight) reads three times:
# each of these was slower there by a factor of 1.5 to 12.
@pytest.mark.parametrize("K, N, s, dtype, calls", [
    (2048, 2048, 0.5, torch.float16, {("columns", 2): "bits", ("columns", 16): "mma", ("offset", 8): "bits", ("offset", 64): "mma"}),
    (2048, 8192, 0.7, torch.float32, {("columns", 1): "bits", ("columns", 8): "mma", ("offset", 16): "mma", ("rows", 4): "bits"}),
    (2048, 8192, 0.7, torch.int8, {("columns", 2): "gather", ("rows", 2): "bits", ("columns", 16): "mma"}),
    (8192, 28672, 0.5, torch.float32, {("rows", 1): "nibble", ("offset", 1): "nibble", ("rows", 2): "nibble", ("rows", 5): "nibble", ("offset", 5): "mma", ("columns", 1): "nibble", ("rows", 64): "mma"})])
def test_cost_model_by_layout(K, N, s, dtype, calls):
    L = _lib.lib()
    L.tllm_set_mma_min_rows(-1)
    rng = np.random.default_rng(16)
    w = random_ternary(rng, K, N, s)
    pw = PackedWeight.from_dense(w)
    Wd = torch.tensor(w, device=dev()).double()
    for (layout, M), kernel in calls.items():
        X = torch.tensor(rng.integers(-4, 5, size=(M, K)), device=dev()).to(dtype)
        x = X.t().contiguous() if layout == "columns" else X
        if layout == "offset":                                        # rows that start on no multiple of 16 bytes
            x = torch.empty(M * K + 1, dtype=dtype, device=dev())[1:].view(M, K).copy_(X)
        counts = lambda: np.array([L.tllm_bits_launch_count(), L.tllm_mma_launch_count(), L.tllm_nibble_launch_count()])
        n0 = counts()
        Y = pw.matmul(x, col_major=layout == "columns", out=torch.empty((M, N), dtype=torch.int32 if dtype == torch.int8 else torch.float32, device=dev()))
        n = counts() - n0
        assert list(n > 0) == [kernel == "bits", kernel == "mma", kernel == "nibble"], (layout, M, kernel, n)
        assert torch.equal(Y.double(), X.double() @ Wd)
    pw.close()


# The price of the register decoder is that of the form it is launched in: shared activations that do not fit are not counted on
@pytest.mark.parametrize("M, K, N, dtype, kernel", [(16, 4888, 13696, torch.float16, "mma"), (14, 4888, 13696, torch.float16, "bits"), (16, 5120, 15360, torch.bfloat16, "mma"), (12, 5120, 15360, torch.bfloat16, "bits"),
                                                    (16, 8192, 10240, torch.bfloat16, "mma"), (8, 8192, 10240, torch.bfloat16, "bits")])
def test_choice_by_the_form_that_is_launched(M, K, N, dtype, kernel):
    L = _lib.lib()
    L.tllm_set_mma_min_rows(-1)
    gen = torch.Generator().manual_seed(K)
    w = torch.randint(-1, 2, (K, N), dtype=torch.int8, generator=gen)
    pw = PackedWeight.from_dense(w.numpy())
    X = torch.randint(-8, 9, (M, K), generator=gen).to(dtype).to(dev())
    b0, m0 = L.tllm_bits_launch_count(), L.tllm_mma_launch_count()
    Y = pw.matmul(X, out=torch.empty((M, N), dtype=torch.float32, device=dev()))
    assert (L.tllm_bits_launch_count() > b0, L.tllm_mma_launch_count() > m0) == (kernel == "bits", kernel == "mma")
    assert torch.equal(Y.double(), X.double() @ w.to(dev()).double())
    pw.close()
