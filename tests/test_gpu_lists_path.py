"""ter_spmm on the reference's arrays with enough rows: the lists are turned into two-bit tiles on the device first
(csrc/lists_kernel.cuh).  Pinned by the oracle's product on the arrays themselves, exact on integers; lists that bit tiles
cannot hold (an entry named twice, a pair that cancels across lists) fall back to the per-column kernel inside the same call."""
import subprocess
import sys

import numpy as np
import pytest
import torch

import oracle
from conftest import ROOT, random_ternary
from ternaryllm_b200 import _lib, ter_spmm

pytestmark = pytest.mark.gpu
DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i8": torch.int8}


def call(x, idx, off, N, K, T, dtype, col_major=False):
    B, M = x.shape[:2]
    X = torch.tensor(x, dtype=DT[dtype], device="cuda")
    if col_major:
        X = X.transpose(1, 2).contiguous()
    ri = torch.tensor(np.asarray(idx).astype(np.int16), device="cuda")
    co = torch.tensor(np.asarray(off).astype(np.int32), device="cuda")
    return ter_spmm.ter_spmm(X, ri, co, None, B, M, N, K, False, False, tile_k=T).double().cpu().numpy()


def kernels():
    L = _lib.lib()
    return np.array([L.tllm_launch_count(), L.tllm_bits_launch_count() + L.tllm_mma_launch_count()])


# one slice, odd slices, tiles of many sizes, several images per block (K > 2048: one row more, a slice more, several more; of tiles that end with
# them and of one that does not), no full tile of columns; each with the fewest rows that are turned into bit tiles (entries * ceil(rows / 4) >= 6e6), and one block of four fewer
@pytest.mark.parametrize("K,N,T,s", [(40, 3, 16, 0.3), (64, 16, 64, 0.5), (200, 130, 64, 0.6), (1000, 70, 256, 0.5), (2048, 300, 256, 0.9), (9000, 40, 512, 0.6),
                                     (8256, 20, 100, 0.5), (2049, 36, 256, 0.5), (2112, 50, 512, 0.6)])
@pytest.mark.parametrize("padding", [0, 4])
def test_exact_on_integer_activations(K, N, T, s, padding):
    rng = np.random.default_rng(K + N)
    w = random_ternary(rng, K, N, s).astype(np.int32)
    idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), T, bool(padding), padding or 4, as_numpy=True)
    least = 4 * (-(-6000000 // (K * N)) - 1) + 1
    for dtype, top in (("f32", 100), ("bf16", 1), ("i8", 127)):
        for B, M in ((1, least), (2, least + 2), (1, least - 1), (3, 3)):
            x = rng.integers(-top, top + 1, size=(B, M, K)).astype(np.float64)
            want = np.stack([oracle.dense_f64(x[b], w.astype(np.int8)) for b in range(B)])
            if dtype == "bf16":
                want = oracle.round_to(want, 2)
            for col_major in (False, True) if M != K else (False,):
                n0 = kernels()
                assert np.array_equal(call(x, idx, off, N, K, T, dtype, col_major), want), (dtype, B, M, col_major)
                launches, products = kernels() - n0
                # converted: the lists, the product (planes before it or not), the per-column kernel for what the tiles cannot hold
                assert (products >= 1 and launches >= products + 2) if M >= least else (products == 0 and launches == 1), (dtype, B, M, col_major)


def converted(x, idx, off, N, K, T):
    n0 = kernels()
    y = call(x, idx, off, N, K, T, "f32")[0]
    assert (kernels() - n0)[1] >= 1
    return y


def test_lists_that_bit_tiles_cannot_hold():
    rng = np.random.default_rng(3)
    K, N, T, M = 512, 64, 64, 800
    w = random_ternary(rng, K, N, 0.5).astype(np.int32)
    idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), T, False, 4, as_numpy=True)
    x = rng.integers(-50, 51, size=(1, M, K)).astype(np.float64)
    o = off.reshape(N, K // T, 4)
    dense = oracle.dense_f64(x[0], w.astype(np.int8))

    def same_as_the_arrays_say(bad, boff=off, differs=True):
        want = oracle.mcsc_product_f64(x[0], bad, boff, N, K, T)
        assert np.array_equal(want, dense) != differs
        assert np.array_equal(converted(x, bad, boff, N, K, T), want)

    for column, tile in ((0, 0), (17, 3), (63, 7)):
        pairs, rest, end = o[column, tile, :3]
        assert pairs + 4 <= rest
        bad = idx.copy()
        bad[pairs] = bad[pairs + 2]                # the first two pairs name the same +1 row
        same_as_the_arrays_say(bad)
        bad = idx.copy()
        bad[pairs + 1] = bad[pairs + 2]            # a row that one pair adds and another takes away
        same_as_the_arrays_say(bad)
        bad = idx.copy()
        bad[pairs + 1] = bad[pairs]                # a pair of one row: nothing
        same_as_the_arrays_say(bad)
    at = np.argwhere((o[:, :, 1] < o[:, :, 2]) & (o[:, :, 0] < o[:, :, 1]))
    for column, tile in at[[0, len(at) // 2, -1]]:
        bad = idx.copy()
        bad[o[column, tile, 1]] = bad[o[column, tile, 0]]      # an entry of a pair again in the remainder
        same_as_the_arrays_say(bad)
        for factor in (2, 0, -3):
            boff = off.reshape(N, K // T, 4).copy()
            boff[column, tile, 3] = factor
            same_as_the_arrays_say(idx, boff.reshape(off.shape))
    same_as_the_arrays_say(idx, differs=False)


GIVEN_BACK = """
import numpy as np, torch
from ternaryllm_b200 import ter_spmm
K, N, T, M = 4096, 8192, 512, 1024                    # 8 MB of tiles, 25 MB of planes
w = np.zeros((K, N), np.int32)
w[::5], w[3::5] = 1, -1
idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), T, False, 4, as_numpy=True)
ri, co = torch.tensor(idx.astype(np.int16), device="cuda"), torch.tensor(off.astype(np.int32), device="cuda")
x, y = torch.ones((1, M, K), device="cuda"), torch.empty((1, M, N), device="cuda")
for _ in range(2):
    ter_spmm.ter_spmm(x, ri, co, None, 1, M, N, K, False, False, tile_k=T, out=y)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    ter_spmm.forget()
    assert torch.cuda.mem_get_info()[0] - held >= 24 << 20, (held, torch.cuda.mem_get_info()[0])
print("ok")
"""


def test_workspaces_are_given_back():
    """Without a handle in the process, forget() with no arguments gives back what the pool of workspaces holds."""
    r = subprocess.run([sys.executable, "-c", GIVEN_BACK], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
