"""The one-launch attention kernels (csrc/attn_kernel.cuh) and the module path that uses them, against the same
attention in fp64.  Bounds: fp32 sums of up to a thousand terms of order one: 1e-5 of the largest output; 16-bit types add the
rounding of the result (eps of it) and of the probabilities (each off by eps of itself at most: eps of the largest value)."""
import pytest
import torch

from ternaryllm_b200 import LlamaTernaryAttention, TernaryConfig, TernaryDecoderLayerTP, _lib

pytestmark = pytest.mark.gpu
DT = {"f32": (torch.float32, 0.0), "f16": (torch.float16, 2.0 ** -11), "bf16": (torch.bfloat16, 2.0 ** -8)}


def reference(qkv, B, M, H, KV, D):
    x = qkv.double().view(B, M, H + 2 * KV, D).transpose(1, 2)
    q, k, v = x[:, :H], x[:, H:H + KV].repeat_interleave(H // KV, 1), x[:, H + KV:].repeat_interleave(H // KV, 1)
    s = q @ k.transpose(2, 3) / D ** 0.5
    s = s.masked_fill(torch.ones(M, M, device=s.device, dtype=torch.bool).triu(1), float("-inf"))
    return (s.softmax(-1) @ v).transpose(1, 2).reshape(B * M, H * D)


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("B,M,H,KV,D", [(1, 1, 4, 4, 64), (1, 31, 4, 1, 64), (2, 32, 8, 2, 128), (1, 33, 4, 2, 64), (3, 100, 2, 1, 128), (1, 257, 8, 8, 64), (2, 64, 4, 1, 128), (1, 65, 4, 4, 128)])
def test_kernel(B, M, H, KV, D, dtype):
    dt, eps = DT[dtype]
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = (torch.randn((B * M, (H + 2 * KV) * D), device="cuda", generator=g) * 2).to(dt)
    y = _lib.binding().causal_attention(qkv, B, M, H, KV, D)
    ref = reference(qkv, B, M, H, KV, D)
    assert float((y.double() - ref).abs().max()) <= (1e-5 + eps) * float(ref.abs().max()) + eps * float(qkv.abs().max())


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("B,H,KV,D,n", [(1, 4, 4, 64, 0), (1, 16, 1, 64, 31), (3, 8, 2, 128, 15), (2, 8, 8, 128, 16), (5, 24, 8, 64, 129), (1, 8, 1, 128, 1023),
                                        (2, 16, 2, 64, 1024), (40, 16, 8, 128, 300)])
def test_decode(B, H, KV, D, n, dtype):
    """Positions 0 .. n, the new one included, at the edges of tiles (32 and 16 keys), of parts (128 keys, up to 8) and of groups."""
    dt, eps = DT[dtype]
    g = torch.Generator(device="cuda").manual_seed(n + B)
    qkv = (torch.randn((B, (H + 2 * KV) * D), device="cuda", generator=g) * 2).to(dt)
    kc, vc = ((torch.randn((B + 1, KV, n + 3, D), device="cuda", generator=g) * 2).to(dt) for _ in range(2))
    wk, wv = kc.clone(), vc.clone()
    wk[:B, :, n], wv[:B, :, n] = qkv[:, H * D:(H + KV) * D].view(B, KV, D), qkv[:, (H + KV) * D:].view(B, KV, D)
    y = _lib.binding().decode_attention(qkv, kc, vc, H, n)
    assert torch.equal(kc, wk) and torch.equal(vc, wv)
    q = qkv[:, :H * D].double().view(B, KV, H // KV, D)
    s = (q @ wk[:B, :, :n + 1].double().transpose(2, 3) / D ** 0.5).softmax(-1)
    ref = (s @ wv[:B, :, :n + 1].double()).reshape(B, H * D)
    assert float((y.double() - ref).abs().max()) <= (1e-5 + eps) * float(ref.abs().max()) + eps * float(wv.abs().max())


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_keys_that_score_minus_infinity(dtype):
    """Finite queries and keys whose product is past the range of fp32: such a key has no weight, also where a row has seen no other
    yet, a whole tile of them or both groups' first tiles.  The fp64 scores of these keys are below the others by 1e39."""
    dt, eps = DT[dtype]
    B, M, H, KV, D, far = 1, 200, 4, 2, 64, 130
    qkv = torch.randn((M, (H + 2 * KV) * D), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(dt)
    qkv[:, 0:H * D:D] = 2.0e19
    qkv[:, H * D:(H + KV) * D:D] = 0
    qkv[:far, H * D:(H + KV) * D:D] = -1.0e20
    y = _lib.binding().causal_attention(qkv, B, M, H, KV, D)
    ref = reference(qkv, B, M, H, KV, D)
    assert float((y[far:].double() - ref[far:]).abs().max()) <= (1e-5 + eps) * float(ref.abs().max()) + eps * float(qkv[:, (H + KV) * D:].abs().max())
    if dtype == "bf16":
        q, rows = 5, 3                                                             # the decode step: 130 such keys, then others
        kc, vc = (torch.randn((rows, KV, M + 1, D), device="cuda", generator=torch.Generator(device="cuda").manual_seed(q)).to(dt) for _ in range(2))
        kc[:, :, :, 0] = 0
        kc[:, :, :far, 0] = -1.0e20
        x = qkv[M - rows:].contiguous()
        got = _lib.binding().decode_attention(x, kc, vc, H, M)
        s = x[:, :H * D].double().view(rows, KV, H // KV, D) @ kc.double().transpose(2, 3) / D ** 0.5
        want = (s.softmax(-1) @ vc.double()).reshape(rows, H * D)
        assert float((got.double() - want).abs().max()) <= (1e-5 + eps) * float(want.abs().max()) + eps * float(vc.abs().max())


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


# many short prompts, which leave most of a tile empty, and longer ones under capture were slower on the library's kernel than on the stock core
@pytest.mark.parametrize("dtype, B, M, captured, own", [("f16", 1, 832, False, True), ("f16", 256, 16, False, False), ("f16", 1, 300, True, True), ("f16", 4, 256, True, False),
                                                        ("f16", 4, 256, False, True), ("f32", 1024, 8, False, False), ("f32", 128, 1, False, True), ("f32", 2, 300, True, True)])
def test_core_of_the_module(dtype, B, M, captured, own):
    dt, eps = DT[dtype]
    cfg = TernaryConfig(hidden_size=2048, num_attention_heads=16, num_key_value_heads=16, sparsity=0.9)
    m = LlamaTernaryAttention(cfg, scales=(0.03,) * 4, generator=torch.Generator().manual_seed(0)).eval()
    x = torch.randn((B, M, 2048), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).to(dt)
    calls, core = [], _lib.binding()
    seen = type("Seen", (), {"matmul": core.matmul, "causal_attention": staticmethod(lambda *a: calls.append(1) or core.causal_attention(*a))})
    with torch.no_grad(), pytest.MonkeyPatch.context() as patch:
        y = m(x)[0]
        patch.setattr(_lib, "binding", lambda: seen)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got = m(x)[0]
            graph.replay()
        else:
            got = m(x)[0]
    assert len(calls) == own
    # either core: probabilities, the core's result and the product's rounded by each
    assert float((got - y).abs().max()) <= (2e-5 + 8 * eps) * float(y.abs().max())


def test_module_under_autocast():
    """The stock core computes in autocast's type and hands that on; so does a prompt that the library's kernel would take."""
    cfg = TernaryConfig(hidden_size=512, num_attention_heads=8, num_key_value_heads=2, sparsity=0.7)
    m = LlamaTernaryAttention(cfg, scales=(0.03,) * 4, generator=torch.Generator().manual_seed(0)).eval()
    x = torch.randn((2, 45, 512), device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.float16):
        y = m(x)[0]
        m._own_core = lambda *a: False
        assert torch.equal(y, m(x)[0]) and y.dtype == torch.float16


def test_layer_with_caches_in_another_order():
    """Caches that are views of another layout (positions first) go to the stock core, as the contiguous ones do to the kernel."""
    layer = TernaryDecoderLayerTP(512, 1024, 8, 8, 64, 0.5, 1, 0, torch.device("cuda"), kv_len=40, max_batch=3, reduce="nccl")
    qkv = torch.randn((3, 24 * 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).bfloat16()
    want = layer.attention(qkv, 3)
    k, v = layer.k_cache, layer.v_cache
    layer.k_cache, layer.v_cache = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v))
    got = layer.attention(qkv, 3)
    assert torch.equal(layer.k_cache, k) and torch.equal(layer.v_cache, v)
    assert float((got - want).abs().max()) <= 4 * 2.0 ** -8 * float(want.abs().max())      # probabilities and results rounded by each


def test_layer_with_a_cache_longer_than_its_length():
    """The layer attends to every position that its caches hold; the one-launch kernel, which stops at the new one, is for caches that end there."""
    layer = TernaryDecoderLayerTP(512, 1024, 8, 8, 64, 0.5, 1, 0, torch.device("cuda"), kv_len=40, max_batch=3, reduce="nccl")
    layer.kv_len = 20
    qkv = torch.randn((3, 24 * 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).bfloat16()
    got = layer.attention(qkv, 3)
    q, k, v = (t.view(3, 8, 64) for t in qkv.split(512, 1))
    assert torch.equal(layer.k_cache[:, :, 20], k) and torch.equal(layer.v_cache[:, :, 20], v)
    s = (layer.k_cache.double() @ q.double()[..., None]).squeeze(-1) / 8
    want = (s.softmax(-1)[:, :, None] @ layer.v_cache.double()).reshape(3, 512)
    # probabilities off by eps of themselves, the result rounded once
    assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * (float(want.abs().max()) + float(layer.v_cache.abs().max()))
