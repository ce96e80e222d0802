"""Which kernel the row-grouped launches of a layer run on, by the launch blocks that a call builds. Runs without a GPU."""
import ctypes as C

import pytest
import torch

from ccfuser_b200 import MoEConfig, MoELayer
from ccfuser_b200 import native as N
from ccfuser_b200.ops import gemm as G


def launches(tokens, d=512, f=2048, experts=16, act="gelu", cf=0.0, native=False, sgd=False):
    """{name: launch block} of one forward and backward pass."""
    from ccfuser_b200.ops.fused import CommContext
    CommContext._instances.clear()
    cfg = MoEConfig(d_model=d, d_ffn=f, num_experts=experts, top_k=2, activation=act, dtype=torch.bfloat16, backend="fused",
                    max_tokens=tokens, capacity_factor=cf or None)
    layer = MoELayer(cfg, device="cpu")
    if sgd:
        layer.fuse_sgd(0.1)
    layer._fused_impl().native_runtime = native
    x = torch.randn(tokens, d).bfloat16().requires_grad_(True)
    with N.record_launches() as rec:
        layer(x).float().sum().backward()
    CommContext._instances.clear()
    if not native:
        blocks = [N.GemmLaunch.from_buffer_copy(c[1][0]) for c in rec.calls if c[0] == "ccf_gemm_launch"]
    else:
        blocks, buf, cnt = [], (N.GemmLaunch * 8)(), C.c_int(0)
        for name, args in rec.calls:
            if name == "ccf_layer_forward":
                assert N.load().ccf_layer_forward(C.byref(N.Layer.from_buffer_copy(args[0])), *args[1:9], None, buf, 8, C.byref(cnt)) == 0
            elif name == "ccf_layer_backward":
                assert N.load().ccf_layer_backward(C.byref(N.Layer.from_buffer_copy(args[0])), *args[1:4],
                                                   C.byref(N.LayerGrads.from_buffer_copy(args[4])), args[5], args[6], None, buf, 8,
                                                   C.byref(cnt)) == 0
            else:
                continue
            blocks += [N.GemmLaunch.from_buffer_copy(bytes(buf[i])) for i in range(cnt.value)]
    out = dict(zip(("gemm1", "gemm2", "dgrad2", "dgrad1"), [b for b in blocks if not b.kgroup]))
    out.update(zip(("wgrad2", "wgrad1"), [b for b in blocks if b.kgroup]))
    return out


def kernel(block):
    return block.few_rows, block.two_cta, block.args.a_rows, block.args.bn


@pytest.mark.parametrize("native", [False, True])
def test_one_cta_kernel_keeps_its_row_bound_and_narrow_tiles(native, monkeypatch):
    """CCFUSER_TWO_CTA=0: with a bound on the rows of every expert the pipeline holds more weights, and a second projection of few
    tiles has narrow ones."""
    monkeypatch.setattr(G, "TWO_CTA_DEFAULT", False)
    got = launches(8, native=native)
    assert [kernel(got[k]) for k in ("gemm1", "gemm2", "dgrad2", "dgrad1")] == [(0, 0, 32, 0), (0, 0, 32, 128), (0, 0, 32, 0), (0, 0, 32, 0)]
    got = launches(400, experts=64, cf=4.0, native=native)      # 50 rows an expert at most, 128 tiles
    assert kernel(got["gemm1"]) == (0, 0, 64, 0) and kernel(got["gemm2"]) == (0, 0, 64, 128)
    got = launches(3000, d=1024, experts=32, native=native)     # no bound, 256 tiles
    assert kernel(got["gemm1"]) == kernel(got["gemm2"]) == (0, 0, 0, 0)


@pytest.mark.parametrize("native", [False, True])
def test_weight_gradients_change_kernels_at_the_measured_rows(native):
    """Plain ones run on gemm_wgrad.cu up to 384 expected rows per expert, in-place ones up to 512, then on CTA pairs."""
    def few(rows, sgd):
        got = launches(rows * 8, d=256, f=512, sgd=sgd, native=native)
        assert all(got[k].two_cta == 1 for k in ("wgrad1", "wgrad2"))
        return [got[k].few_rows for k in ("wgrad1", "wgrad2")]
    assert few(384, False) == [1, 1] and few(385, False) == [0, 0]
    assert few(512, True) == [1, 1] and few(513, True) == [0, 0]
