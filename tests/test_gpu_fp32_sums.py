"""fp32 activations: sums over a long K stay as good as fp32 additions rounded to nearest, 2^-23 of the result (2-norm of the error
against fp64 over 2-norm of the result; the kernels on index lists and the four-bit planes are at 5e-8 to 1.1e-7 on the same data).
Of the kernels on bit tiles this asks that the tensor core, which cuts bits off its running sum toward zero, never holds a
sum for long: values of one sign show the bias of that, and a few large values among small ones the bits that are cut."""
import numpy as np
import pytest
import torch

from conftest import random_ternary
from ternaryllm_b200 import PackedMLP, PackedWeight

pytestmark = pytest.mark.gpu


def error(got, want):
    return float((got.double() - want).norm() / want.norm())


# 512 and 256 rows: whole tiles of the batched kernel; 64: units of a tile shared by blocks or a cluster; 8: decoded in registers
@pytest.mark.parametrize("M", [512, 256, 64, 8])
@pytest.mark.parametrize("K,N,data", [(6912, 2560, "gated"), (5120, 2048, "positive"), (8192, 1024, "normal")])
def test_product(K, N, M, data):
    g = torch.Generator(device="cuda").manual_seed(K + M)
    a, b = (torch.randn((M, K), device="cuda", generator=g) for _ in range(2))
    x = {"gated": a * torch.sigmoid(a) * b, "positive": torch.rand((M, K), device="cuda", generator=g), "normal": a}[data]
    w = np.ones((K, N), np.int8) if data == "positive" else random_ternary(np.random.default_rng(K), K, N, 0.5)
    pw = PackedWeight.from_dense(w)
    assert error(pw.matmul(x), x.double() @ torch.tensor(w, device="cuda").double()) <= 2.0 ** -23
    pw.close()


@pytest.mark.parametrize("M", [8, 16, 256])
def test_gated_intermediate_result(M):
    hidden, inter = 2560, 6912
    rng = np.random.default_rng(7)
    ws = [random_ternary(rng, *shape, 0.5) for shape in ((hidden, inter), (hidden, inter), (inter, hidden))]
    mlp = PackedMLP(*ws, 0.0371, 0.0293, 0.03125)
    x = torch.randn((M, hidden), device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    gate, up = (x.double() @ torch.tensor(w, device="cuda").double() * s for w, s in ((ws[0], 0.0371), (ws[1], 0.0293)))
    h = torch.empty((M, inter), device="cuda")
    mlp.forward(x, h=h)
    assert error(h, gate * torch.sigmoid(gate) * up) <= 2.0 ** -23
    mlp.close()
