"""A call that takes a workspace may be the first of its process and be made under stream capture: the pool the workspaces come
from is made there and then.  Each case in a process of its own; the graph's result is exact on integers, twice."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
import numpy as np, torch
from ternaryllm_b200 import PackedWeight, ter_spmm
kind, K, N, M = sys.argv[1], 1024, 2048, 64
rng = np.random.default_rng(0)
w = rng.integers(-1, 2, size=(K, N)).astype(np.int8)
x = torch.tensor(rng.integers(-9, 10, size=(M, K)), dtype=torch.int8 if kind == "i8" else torch.float32, device="cuda")
if kind == "lists":
    wi, T = w.astype(np.int32), ter_spmm.tile_size_for(K)
    idx, off, _ = ter_spmm.convert_to_ter_tiled_mcsc(wi, N, K, int((wi == 1).sum()), int((wi == -1).sum()), T, False, 4, as_numpy=True)
    ri, co = torch.tensor(idx.astype(np.int16), device="cuda"), torch.tensor(off.astype(np.int32), device="cuda")
    call = lambda: ter_spmm.ter_spmm(x.view(1, M, K), ri, co, None, 1, M, N, K, False, False)[0]
else:
    pw = PackedWeight.from_dense(w)
    call = lambda: pw.matmul(x)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = call()
want = x.double() @ torch.tensor(w, device="cuda").double()
for _ in range(2):
    y.zero_()
    graph.replay()
    assert torch.equal(y.double(), want)
assert torch.equal(call().double(), want)
print("ok")
"""


@pytest.mark.parametrize("kind", ["f32", "i8", "lists"])
def test_first_call_under_capture(kind):
    r = subprocess.run([sys.executable, "-c", PROGRAM, kind], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
