"""Residual add + RMSNorm behind a kernel that lets it start early: every buffer it reads, the norm weight included, may be
that kernel's result.  fp32 throughout: sums of 2048 squares and one product, 1e-5 of the largest output."""
import numpy as np
import pytest
import torch

from conftest import random_ternary
from ternaryllm_b200 import PackedWeight
from ternaryllm_b200.tensor_parallel import PeerReduce, add_rms_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("peer", [False, True])
@pytest.mark.parametrize("rows", [1, 40])
def test_weight_made_by_the_preceding_product(rows, peer):
    K, hidden = 4096, 2048
    w = random_ternary(np.random.default_rng(2), K, hidden, 0.5)
    pw = PackedWeight.from_dense(w, scale=0.0625)
    Wd = torch.tensor(w, device="cuda").double() * 0.0625
    reduce = PeerReduce(rows, hidden, "cuda") if peer else None
    gain = torch.zeros((1, hidden), device="cuda")
    out = torch.empty((rows, hidden), device="cuda")
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x, delta = (torch.randn((rows, hidden), device="cuda", generator=g) for _ in range(2))
        a = torch.randn((1, K), device="cuda", generator=g)
        want_x = x + delta
        torch.cuda.synchronize()
        pw.matmul(a, out=gain)
        got = reduce.reduce(delta, x, out=out, weight=gain) if peer else add_rms_norm(x, delta, out=out, weight=gain)
        v = want_x.double()
        want = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6) * (a.double() @ Wd)
        assert torch.equal(x, want_x)
        assert float((got.double() - want).abs().max()) <= 1e-5 * float(want.abs().max()), seed
    if peer:
        reduce.close()
    pw.close()
