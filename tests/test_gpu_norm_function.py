"""LayerNorm's autograd function (csrc/torch_norm.cpp): what autograd asks of a function, and the forward kernel's walk over rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# bf16 results of sums in fp32: half a unit in the last place of the largest value, 2^-9, and as much for the rounded inputs' products
TOL = 2.0 ** -8


def _ref(x, w, b, gy, eps=1e-5):
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    bd = None if b is None else b.detach().double().requires_grad_(True)
    y = torch.nn.functional.layer_norm(xd, (x.shape[-1],), wd, bd, eps)
    y.backward(gy.double())
    return y, xd.grad, wd.grad, None if b is None else bd.grad


def _close(a, r):
    assert a.shape == r.shape
    assert float((a.double() - r).abs().max() / r.abs().max().clamp_min(1e-6)) < TOL


# one row, one block, one row more than the grid's warps take at once (2 blocks of 8 rows on each of 148 SMs), several rows per warp
@pytest.mark.parametrize("rows", [1, 8, 2369, 2368 * 3 + 5])
@pytest.mark.parametrize("d", [8, 264, 768, 2048])
def test_rows_per_warp(rows, d):
    from ccfuser_b200.ops.norm import layer_norm
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + d)
    x = torch.randn(rows, d, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (1 + 0.2 * torch.randn(d, generator=g, device="cuda")).bfloat16().requires_grad_(True)
    b = (0.1 * torch.randn(d, generator=g, device="cuda")).bfloat16().requires_grad_(True)
    gy = torch.randn(rows, d, generator=g, device="cuda").bfloat16()
    y = layer_norm(x, (d,), w, b)
    y.backward(gy)
    ry, rx, rw, rb = _ref(x, w, b, gy)
    _close(y, ry)
    _close(x.grad, rx)
    _close(w.grad, rw)
    _close(b.grad, rb)


def test_strided_inputs_saved_tensor_hooks_and_frozen_weights():
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops.norm import layer_norm
    torch.manual_seed(5)
    base = torch.randn(4, 50, 96, device="cuda").bfloat16()
    x = base.transpose(0, 1)[:, :, ::2].detach().requires_grad_(True)        # no stride of a contiguous tensor
    w = torch.randn(48, device="cuda").bfloat16()                            # needs no gradient
    gy = torch.randn(48, 50, 4, device="cuda").bfloat16().permute(1, 2, 0)
    packed = []
    before = N.LAUNCHES[0]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
        y = layer_norm(x, (48,), w, None)
    y.backward(gy)
    assert len(packed) == 4 and N.LAUNCHES[0] - before == 3
    assert w.grad is None
    ry, rx, _, _ = _ref(x, w, None, gy)
    _close(y, ry)
    _close(x.grad, rx)


def test_transforms_are_refused():
    from ccfuser_b200.ops.norm import layer_norm
    x, w = torch.randn(4, 3, 64, device="cuda").bfloat16(), torch.ones(64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: layer_norm(t, (64,), w, None))(x)
    import torch.autograd.forward_ad as fwd
    with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        layer_norm(fwd.make_dual(x, torch.ones_like(x)), (64,), w, None)


@pytest.mark.parametrize("bias", [True, False])
def test_a_traced_graph_replays_the_kernels(bias):
    """torch.jit.trace records the operation, not only the allocation of its output: on another input the graph gives what the module
    gives, forward and backward, to the bit."""
    from ccfuser_b200.ops.norm import LayerNorm
    torch.manual_seed(11)
    norm = LayerNorm(768, bias=bias, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        for p in norm.parameters():
            p.normal_()
    x, x2, gy = (torch.randn(5, 31, 768, device="cuda").bfloat16() for _ in range(3))
    traced = torch.jit.trace(norm, (x,), check_trace=False)

    def run(f):
        v = x2.clone().requires_grad_(True)
        norm.zero_grad()
        # what an allocation finds is not an earlier result
        junk = [torch.full_like(x, 3.0) for _ in range(8)]
        del junk
        y = f(v)
        y.backward(gy)
        return [y.detach(), v.grad] + [p.grad.clone() for p in norm.parameters()]
    for a, b in zip(run(traced), run(norm)):
        assert torch.equal(a, b)


def test_without_the_module_the_kernels_run_from_python(monkeypatch):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops.norm import LayerNorm
    torch.manual_seed(13)
    norm = LayerNorm(264, device="cuda", dtype=torch.float16)
    x, gy = (torch.randn(37, 264, device="cuda").half() for _ in range(2))

    def run():
        v = x.clone().requires_grad_(True)
        norm.zero_grad()
        before = N.LAUNCHES[0]
        norm(v).backward(gy)
        assert N.LAUNCHES[0] - before == 3
        return [v.grad] + [p.grad.clone() for p in norm.parameters()]
    want = run()
    monkeypatch.setattr(N, "_torch_module", None)
    monkeypatch.setattr(N, "_torch_module_tried", True)
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
