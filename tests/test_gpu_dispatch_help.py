"""Epilogue warps that push rows until their first accumulator is due (needs a B200): every row arrives once, whoever pushes it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows = 2 * tokens, on both sides of what the dedicated warps hold (592 with 148 SMs) and of the change of chunk size (4096); few experts
# run on CTA pairs, many on the kernel for few rows
@pytest.mark.parametrize("tokens", [1, 296, 297, 2048, 2049, 3001])
@pytest.mark.parametrize("experts", [2, 16])
@pytest.mark.parametrize("act", ["gelu", "swiglu"])
def test_rows_pushed_with_help_are_the_rows_pushed_without(tokens, experts, act, monkeypatch):
    """The epilogue warps alone (comm_warps = 0) against dedicated warps with help: outputs and gradients of the same bits."""
    from ccfuser_b200 import MoEConfig, MoELayer
    from ccfuser_b200.ops import gemm as G
    got = []
    for dedicated in (0, 1):
        monkeypatch.setattr(G, "COMM_WARPS_DEFAULT", dedicated)
        torch.manual_seed(7)
        cfg = MoEConfig(d_model=384, d_ffn=512, num_experts=experts, top_k=2, activation=act, dtype=torch.bfloat16, backend="fused",
                        max_tokens=tokens)
        layer = MoELayer(cfg, device="cuda")
        x = torch.randn(tokens, 384, device="cuda").bfloat16().requires_grad_(True)
        dy = torch.randn(tokens, 384, device="cuda").bfloat16()
        for _ in range(2):
            x.grad = None
            layer.zero_grad()
            y = layer(x)
            y.backward(dy)
        layer.check_status()
        got.append([y.detach().clone(), x.grad] + [p.grad for p in layer.parameters()])
        layer.release()
    for a, b in zip(*got):
        assert torch.equal(a, b)
