"""Ranks choose their kernels from their own number of tokens; the completion count that one rank sends per row is the one that the
other expects. Host side, without a GPU: 2 gloo ranks whose calls lie on both sides of the kernels' limits."""
import pytest
import torch

from tests.mp_util import run_ranks

D = 320


def _units(rank, world, tokens, native):
    from ccfuser_b200 import MoEConfig, MoELayer
    from ccfuser_b200 import native as N
    cfg = MoEConfig(d_model=D, d_ffn=256, num_experts=4, top_k=2, activation="gelu", dtype=torch.bfloat16, ep_size=world,
                    backend="fused", max_tokens=max(tokens))
    layer = MoELayer(cfg, device="cpu")
    fm = layer._fused_impl()
    fm.native_runtime = native
    x = torch.randn(tokens[rank], D).bfloat16().requires_grad_(True)
    with N.record_launches() as rec:
        layer(x).float().sum().backward()
    return [c[1][3] for c in rec.calls if c[0] == "ccf_combine_wait"]


@pytest.mark.parametrize("tokens", [(3000, 10), (10, 3000), (1, 200)])
def test_ranks_of_one_call_expect_the_same_units(tokens):
    got = run_ranks(_units, 2, tokens, False)
    assert got == [[D // 32] * 2] * 2        # forward and backward, on both ranks


def test_the_unit_has_no_kernel_in_it():
    from ccfuser_b200.ops import gemm as G
    for n in (64, 96, 256, 320, 2048, 4096):
        assert G.combine_units(n) == G.combine_units(n, few_rows=True) == n // 32
