"""Views that begin off a 16-byte boundary are copied before a kernel reads them: the same results as from aligned tensors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t):
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    v = buf[3:3 + t.numel()].view(t.shape)
    v.copy_(t)
    assert v.data_ptr() % 16 != 0 and v.is_contiguous()
    return v


@pytest.mark.parametrize("python", [False, True])
def test_layer_norm(python, monkeypatch):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops.norm import layer_norm
    N.torch_module()
    if python:
        monkeypatch.setattr(N, "_torch_module", None)
    torch.manual_seed(2)
    x, gy = (torch.randn(19, 768, device="cuda").bfloat16() for _ in range(2))
    w, b = (torch.randn(768, device="cuda").bfloat16() for _ in range(2))

    def run(*t):
        v, wv, bv = (p.detach().requires_grad_(True) for p in t[:3])
        y = layer_norm(v, (768,), wv, bv)
        y.backward(t[3])
        return y.detach(), v.grad, wv.grad, bv.grad
    want = run(x, w, b, gy)
    for i in range(4):
        args = [_off(t) if i == j else t for j, t in enumerate((x, w, b, gy))]
        for a, r in zip(run(*args), want):
            assert torch.equal(a, r)


@pytest.mark.parametrize("native", [True, False])
def test_upstream_gradient_of_a_layer(native):
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(4)
    layer = MoELayer(MoEConfig(d_model=256, d_ffn=512, num_experts=8, top_k=2, dtype=torch.bfloat16, backend="fused", max_tokens=300),
                     device="cuda")
    layer._fused_impl().native_runtime = native
    x, dy = (torch.randn(300, 256, device="cuda").bfloat16() for _ in range(2))

    def run(g):
        v = x.clone().requires_grad_(True)
        layer.zero_grad()
        layer(v).backward(g)
        return [v.grad] + [p.grad for p in layer.parameters()]
    want = run(dy)
    for a, r in zip(run(_off(dy)), want):
        assert torch.equal(a, r)
    layer.check_status()
    layer.release()
