"""A layer's results do not depend on the kernels that its launches run on: all sum over k in order and share their arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pass(cfg, tokens, seed=3):
    from ccfuser_b200 import MoELayer
    torch.manual_seed(seed)
    layer = MoELayer(cfg, device="cuda")
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0, 0.05)
    x, dy = (torch.randn(tokens, cfg.d_model, device="cuda").to(cfg.dtype) for _ in range(2))
    x.requires_grad_(True)
    y = layer(x)
    y.backward(dy)
    layer.check_status()
    out = [y.detach(), x.grad] + [p.grad for p in layer.parameters()]
    layer.release()
    return out


# 8, 100, 200, 300, 500 rows an expert: below and above every limit of the rule, and a small capacity
@pytest.mark.parametrize("tokens,cf", [(32, 0.0), (32, 1.5), (400, 0.0), (800, 0.0), (1200, 0.0), (2000, 0.0)])
@pytest.mark.parametrize("act,dtype", [("gelu", torch.bfloat16), ("swiglu", torch.float16)])
def test_same_bits_on_every_kernel(tokens, cf, act, dtype, monkeypatch):
    from ccfuser_b200 import MoEConfig
    from ccfuser_b200.ops import gemm as G
    cfg = MoEConfig(d_model=256, d_ffn=512, num_experts=8, top_k=2, activation=act, dtype=dtype, backend="fused", max_tokens=tokens,
                    capacity_factor=cf or None)
    want = _pass(cfg, tokens)
    for two_cta, small in ((True, -1), (True, 1 << 20), (False, 320)):
        monkeypatch.setattr(G, "TWO_CTA_DEFAULT", two_cta)
        monkeypatch.setattr(G, "SMALL_ROWS_DEFAULT", small)
        for a, b in zip(_pass(cfg, tokens), want):
            assert torch.equal(a, b)
