"""install(auto_prepare=True): a call repacks its arrays only after everything about it has been checked.  A refused call must
leave no packed copy behind (a later tensor at the same address would get it) and must not read arrays of the wrong size."""
import types

import numpy as np
import pytest
import torch

import oracle
from conftest import random_ternary
from ternaryllm_b200 import _lib, ter_spmm


@pytest.fixture
def auto(monkeypatch):
    monkeypatch.setattr(ter_spmm, "AUTO_PREPARE", True)
    yield
    if torch.cuda.is_available():
        ter_spmm.forget()


def test_nothing_is_repacked_for_a_refused_call(auto, monkeypatch):
    seen = []
    monkeypatch.setattr(ter_spmm, "prepare", lambda *a: seen.append(a))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    fake = types.SimpleNamespace(is_cuda=True)
    with pytest.raises(RuntimeError):
        ter_spmm.ter_spmm(fake, fake, fake, None, 1, 4, 8, 16, False, False)
    assert not seen


@pytest.mark.gpu
def test_checks_come_before_the_copy(auto):
    rng = np.random.default_rng(4)
    K, N, T, M = 512, 96, 128, 6
    w = random_ternary(rng, K, N, 0.5).astype(np.int32)
    idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(w, N, K, int((w == 1).sum()), int((w == -1).sum()), T, False, 4, as_numpy=True)
    ri, co = torch.tensor(idx.astype(np.int16), device="cuda"), torch.tensor(off.astype(np.int32), device="cuda")
    x = rng.integers(-9, 10, size=(1, M, K)).astype(np.float64)
    X = torch.tensor(x, dtype=torch.float32, device="cuda")
    args = (1, M, N, K, False, False)
    for call in (lambda: ter_spmm.ter_spmm(X, ri.int(), co, None, *args, tile_k=T),                 # ids of another type
                 lambda: ter_spmm.ter_spmm(X, ri, co.long(), None, *args, tile_k=T),
                 lambda: ter_spmm.ter_spmm(X, ri, co[:-4], None, *args, tile_k=T),                  # offsets of one list missing
                 lambda: ter_spmm.ter_spmm(X.double(), ri, co, None, *args, tile_k=T),
                 lambda: ter_spmm.ter_spmm(X[:, :, :-1], ri, co, None, *args, tile_k=T),
                 lambda: ter_spmm.ter_spmm(X, ri, co, None, *args, tile_k=T, out=torch.empty((1, M, N), device="cuda", dtype=torch.float16))):
        with pytest.raises(RuntimeError, match="ter_spmm"):
            call()
        assert ter_spmm.forget() == 0
    assert ter_spmm.ter_spmm(X[:0], ri, co, None, 0, M, N, K, False, False, tile_k=T).shape == (0, M, N) and ter_spmm.forget() == 0
    n0 = _lib.lib().tllm_launch_count()
    for _ in range(2):
        y = ter_spmm.ter_spmm(X, ri, co, None, *args, tile_k=T, scale=0.5)
        assert np.array_equal(y[0].double().cpu().numpy(), oracle.dense_f64(x[0], w.astype(np.int8), 0.5))
    assert _lib.lib().tllm_launch_count() > n0 and ter_spmm.forget(ri, co) == 1 and ter_spmm.forget() == 0
    # under capture nothing is repacked: the per-column kernel or the conversion is what gets recorded
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = ter_spmm.ter_spmm(X, ri, co, None, *args, tile_k=T)
    graph.replay()
    assert np.array_equal(y[0].double().cpu().numpy(), oracle.dense_f64(x[0], w.astype(np.int8))) and ter_spmm.forget() == 0
