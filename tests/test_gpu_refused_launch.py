"""A layer call one of whose later launches is refused raises, and the next call is not affected by it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off_boundary(p):
    """The same values two bytes off a 16-byte boundary: the tensor map of a launch that reads them cannot be encoded."""
    buf = torch.empty(p.numel() + 8, dtype=p.dtype, device=p.device)
    v = buf[1:1 + p.numel()].view(p.shape)
    v.copy_(p)
    return v


# the weight that is off a boundary, and the first launch that reads it: GEMM-2 (after dispatch + GEMM-1), or dgrad-1 (after the
# dy dispatch, dgrad-2 and, without the in-place SGD, the weight gradients)
@pytest.mark.parametrize("act,tokens,where,sgd", [("gelu", 300, "forward", False), ("swiglu", 40, "forward", False),
                                                  ("gelu", 3000, "backward", False), ("swiglu", 300, "backward", False),
                                                  ("relu", 40, "backward", True)])
def test_call_after_a_refused_launch(act, tokens, where, sgd):
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(tokens)
    cfg = MoEConfig(d_model=256, d_ffn=512, num_experts=8, top_k=2, activation=act, dtype=torch.bfloat16, backend="fused",
                    max_tokens=tokens)
    layer = MoELayer(cfg, device="cuda")
    fm, params = layer._fused_impl(), list(layer.parameters())
    x, x2 = (torch.randn(tokens, 256, device="cuda", dtype=torch.bfloat16).requires_grad_() for _ in range(2))
    gy = torch.randn_like(x)

    def step(inp):
        for p in (inp, *params):
            p.grad = None
        y = layer(inp)
        y.backward(gy)
        return [y.detach(), *(p.grad for p in (inp, *params) if p.grad is not None)]
    want = step(x2)
    if sgd:
        layer.fuse_sgd(0.5)
    bad = layer.experts.h4toh.weight if where == "forward" else layer.experts.htoh4.weight
    good, before = bad.data, [p.detach().clone() for p in params]
    if where == "forward":
        bad.data = _off_boundary(good)
        with torch.no_grad(), pytest.raises(RuntimeError):
            layer(x)
    else:
        y = layer(x)
        bad.data = _off_boundary(good)
        with pytest.raises(RuntimeError):
            y.backward(gy)
        del y
    bad.data = good
    torch.cuda.synchronize()
    assert not fm.ctx.tile_flags.any()      # no tile of the next call may pass its gate before its rows have arrived
    if sgd:
        layer.fuse_sgd(None)
        with torch.no_grad():
            for p, v in zip(params, before):
                p.copy_(v)
    for a, b in zip(step(x2), want):
        assert torch.equal(a, b)
    layer.check_status()
    layer.release()


def test_call_after_a_backward_pass_that_has_no_kernel():
    """d_model 64 runs forward only: its backward pass is refused at the weight gradient, after the dispatch of the gradients."""
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(3)
    cfg = MoEConfig(d_model=64, d_ffn=128, num_experts=8, top_k=2, dtype=torch.bfloat16, backend="fused", max_tokens=2000)
    layer = MoELayer(cfg, device="cuda")
    x, x2 = (torch.randn(2000, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    with torch.no_grad():
        want = layer(x2)
    y = layer(x)
    with pytest.raises(RuntimeError):
        y.backward(torch.randn_like(x))
    torch.cuda.synchronize()
    assert not layer._fused_impl().ctx.tile_flags.any()
    with torch.no_grad():
        assert torch.equal(layer(x2), want)
    layer.check_status()
    layer.release()
