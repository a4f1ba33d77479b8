"""The buffer between an MLP handle's two products outlives every call: a graph captured with it is replayed after a host-buffer
call with more rows than it holds."""
import numpy as np
import pytest
import torch

import oracle
from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, _lib

pytestmark = pytest.mark.gpu


def test_graph_replayed_after_a_larger_host_call():
    rng = np.random.default_rng(9)
    hidden, inter = 512, 1376
    ws = [random_ternary(rng, *shape, 0.6) for shape in ((hidden, inter), (hidden, inter), (inter, hidden))]
    mlp = PackedMLP(*ws, 0.02, 0.03, 0.04)
    x = torch.randn((24, hidden), device="cuda").half()
    want = mlp.forward(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = mlp.forward(x)
    host = rng.standard_normal((400, hidden)).astype(np.float32)
    ref = oracle.mlp_f64(host.astype(np.float64), *ws, 0.02, 0.03, 0.04, h_round=3)
    h = np.empty((400, inter), np.float32)
    _lib.check(_lib.lib().tllm_mlp_forward_host(mlp._h, _lib.np_ptr(host), _lib.F32, _lib.ROW_MAJOR, 400, _lib.np_ptr(h)))
    assert np.max(np.abs(host - ref)) <= 1e-5 * np.max(np.abs(ref)) and np.isfinite(h).all()
    junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(8)]      # whatever was given back is used again
    y.zero_()
    graph.replay()
    assert torch.equal(y, want) and len(junk) == 8
    mlp.close()
