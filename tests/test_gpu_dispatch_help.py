"""Epilogue warps that push rows until their first accumulator is due: when they help, and (on a B200) that every row arrives once,
whoever pushes it."""
import pytest
import torch


@pytest.mark.parametrize("pushing", [1, 8, 100, 148, 1 << 20])
def test_help_begins_where_a_dedicated_warp_has_more_than_one_chunk(pushing):
    """Chunks have two rows up to 4096 rows in all; two dedicated warps push in each of the first ``pushing`` CTAs of 148."""
    from ccfuser_b200 import native as N
    helps = N.load().ccf_dispatch_help
    warps = 2 * min(pushing, 148)
    for pair in (0, 1):
        for kept in (0, 1, 2 * warps - 1, 2 * warps, 2 * warps + 1, 2 * warps + 2, 4096):
            assert helps(kept, pushing, 148, pair) == int((kept + 1) // 2 > warps), kept
        assert helps(4097, pushing, 148, pair) == helps(1 << 20, pushing, 148, pair) == pair


# rows = 2 * tokens, on both sides of what the dedicated warps hold (592 with 148 SMs) and of the change of chunk size (4096); few experts
# run on CTA pairs, many on the kernel for few rows
@pytest.mark.gpu
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


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [9, 40, 296, 2049])
@pytest.mark.parametrize("experts", [2, 16])
def test_rows_pushed_by_a_few_ctas_are_the_rows_pushed_by_all(tokens, experts):
    """Eight CTAs whose dedicated warps push, with help from 33 rows on, against all."""
    from ccfuser_b200 import MoEConfig, MoELayer
    got = []
    for ctas in (1 << 20, 8):
        torch.manual_seed(7)
        cfg = MoEConfig(d_model=384, d_ffn=512, num_experts=experts, top_k=2, activation="gelu", dtype=torch.bfloat16, backend="fused",
                        max_tokens=tokens)
        layer = MoELayer(cfg, device="cuda")
        context = layer._fused_impl().ctx
        before, context.n_comm = context.n_comm, ctas
        try:
            x = torch.randn(tokens, 384, device="cuda").bfloat16().requires_grad_(True)
            dy = torch.randn(tokens, 384, device="cuda").bfloat16()
            for _ in range(2):
                x.grad = None
                layer.zero_grad()
                y = layer(x)
                y.backward(dy)
            layer.check_status()
            got.append([y.detach().clone(), x.grad] + [p.grad for p in layer.parameters()])
        finally:
            context.n_comm = before
        layer.release()
    for a, b in zip(*got):
        assert torch.equal(a, b)
