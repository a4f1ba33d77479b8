"""The one-launch causal attention (csrc/attn_kernel.cuh) and the module path that uses it, against the same attention in fp64.
Bounds: fp32 arithmetic on values of order one, sums of up to a few hundred terms: 1e-5 of the largest output; 16-bit types add
the rounding of the result (eps)."""
import pytest
import torch

from ternaryllm_b200 import LlamaTernaryAttention, TernaryConfig, _lib

pytestmark = pytest.mark.gpu
DT = {"f32": (torch.float32, 0.0), "f16": (torch.float16, 2.0 ** -11), "bf16": (torch.bfloat16, 2.0 ** -8)}


def reference(qkv, B, M, H, KV, D):
    x = qkv.double().view(B, M, H + 2 * KV, D).transpose(1, 2)
    q, k, v = x[:, :H], x[:, H:H + KV].repeat_interleave(H // KV, 1), x[:, H + KV:].repeat_interleave(H // KV, 1)
    s = q @ k.transpose(2, 3) / D ** 0.5
    s = s.masked_fill(torch.ones(M, M, device=s.device, dtype=torch.bool).triu(1), float("-inf"))
    return (s.softmax(-1) @ v).transpose(1, 2).reshape(B * M, H * D)


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("B,M,H,KV,D", [(1, 1, 4, 4, 64), (1, 31, 4, 1, 64), (2, 32, 8, 2, 128), (1, 33, 4, 2, 64), (3, 100, 2, 1, 128), (1, 257, 8, 8, 64)])
def test_kernel(B, M, H, KV, D, dtype):
    dt, eps = DT[dtype]
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = (torch.randn((B * M, (H + 2 * KV) * D), device="cuda", generator=g) * 2).to(dt)
    y = _lib.binding().causal_attention(qkv, B, M, H, KV, D)
    ref = reference(qkv, B, M, H, KV, D)
    assert float((y.double() - ref).abs().max()) <= (1e-5 + eps) * float(ref.abs().max())


@pytest.mark.parametrize("dtype", list(DT))
def test_module_agrees_with_the_stock_core(dtype):
    dt, eps = DT[dtype]
    cfg = TernaryConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, sparsity=0.7)
    m = LlamaTernaryAttention(cfg, scales=(0.03,) * 4, generator=torch.Generator().manual_seed(0)).eval()
    x = torch.randn((2, 45, 512), device="cuda").to(dt)
    with torch.no_grad():
        own = m(x)[0]
        m._own_core = lambda *a: False
        stock = m(x)[0]
    # 16-bit: the stock core rounds its probabilities and the two products round q | k | v and the result
    assert float((own - stock).abs().max()) <= (2e-5 + 8 * eps) * float(stock.abs().max())
