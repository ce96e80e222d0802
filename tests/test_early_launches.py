"""Launches of small calls that are set up while the kernel in front of them still runs (csrc/sm100.cuh): the order that every kernel
with tensor memory keeps, and on a B200 the same results as with launches one after the other."""
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ccfuser_b200", "csrc")


@pytest.mark.parametrize("name", ["router.cu", "gemm2.cu", "gemm_swap.cu", "gemm_wgrad.cu"])
def test_tensor_memory_is_taken_behind_the_wait_and_before_the_next_kernel_is_let_in(name):
    """A kernel that held columns while it waits could keep them from the kernel that it waits for; one that let the next kernel in before
    it has its columns could wait for that one."""
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    body = code[code.index("__global__"):]
    steps = [m.group(1) for m in re.finditer(r"\b(wait_for_previous|tmem_alloc(?:_pair)?|__syncthreads|let_next_in|after_previous)\(", body)]
    steps = ["tmem_alloc" if s.startswith("tmem_alloc") else s for s in steps]
    assert steps[:4] == ["wait_for_previous", "tmem_alloc", "__syncthreads", "let_next_in"], steps[:6]
    assert "after_previous" not in steps and steps.count("let_next_in") == 1 == steps.count("tmem_alloc")


def _layer(act, experts, tokens, sgd):
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(5)
    cfg = MoEConfig(d_model=256, d_ffn=512, num_experts=experts, top_k=2, activation=act, dtype=torch.bfloat16, backend="fused", max_tokens=tokens)
    layer = MoELayer(cfg, device="cuda")
    if sgd:
        layer.fuse_sgd(0.05)
    layer._fused_impl().ctx.use_device_epoch()
    return layer


# rows of an expert on both sides of the change to CTA pairs (320) and of the weight gradients' (384 and 512); all below 4096 slots
@pytest.mark.gpu
@pytest.mark.parametrize("act", ["gelu", "swiglu"])
@pytest.mark.parametrize("experts,tokens", [(8, 16), (8, 301), (2, 333), (2, 600)])
@pytest.mark.parametrize("sgd", [False, True])
def test_passes_with_and_without_early_launches_agree(act, experts, tokens, sgd):
    """Training passes, the last with an inference call right behind it (with ``sgd`` behind an update of its weights in place): eager, where
    launches overlap, against a replayed graph, where they do not."""
    from ccfuser_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(9)
    mk = lambda: torch.randn(tokens, 256, device="cuda", generator=g).bfloat16()  # noqa: E731
    xs, dys = [mk() for _ in range(4)], [mk() for _ in range(4)]
    got = []
    for graphed in (False, True):
        layer = _layer(act, experts, tokens, sgd)
        before = [p.detach().clone() for p in layer.parameters()]
        x, dy = torch.empty_like(xs[0]).requires_grad_(True), torch.empty_like(dys[0])

        def one():
            x.grad = None
            for p in layer.parameters():
                p.grad = None
            y = layer(x)
            y.backward(dy)
            with torch.no_grad():
                z = layer(x)
            return [y.detach(), z, x.grad] + [p.grad for p in layer.parameters() if p.grad is not None]

        def load(i):
            with torch.no_grad():
                x.copy_(xs[i])
                dy.copy_(dys[i])

        load(0)
        if graphed:
            ws = G.Workspace.get("cuda")
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            ws.ordered_after()
            with torch.cuda.stream(side):
                one()                                  # first use sets the kernels up outside the capture
            torch.cuda.synchronize()
            ws.ordered_after()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                outs = one()
            torch.cuda.synchronize()
            ws.ordered_after()
            with torch.no_grad():
                for p, b in zip(layer.parameters(), before):
                    p.copy_(b)
        kept = []
        for i in range(4):
            load(i)
            if graphed:
                graph.replay()
            else:
                outs = one()
            kept.append([t.clone() for t in outs])
        kept.append([p.detach().clone() for p in layer.parameters()])
        layer.check_status()
        got.append(kept)
        if graphed:
            del graph, outs
        layer.release()
    for a, b in zip(*got):
        assert len(a) == len(b)
        for s, t in zip(a, b):
            assert torch.equal(s, t)
    if sgd:
        assert any(not torch.equal(p, b) for p, b in zip(got[0][-1], before))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,d,experts", [(1, 64, 256), (128, 64, 256), (2000, 64, 256), (300, 1024, 64), (4096, 128, 200)])
def test_routers_right_behind_each_other(tokens, d, experts):
    """Kernels with tensor memory and little shared memory, which lie side by side on an SM: 64 in a row against one at a time."""
    from ccfuser_b200.ops import router as R
    g = torch.Generator(device="cuda").manual_seed(2)
    ws = [torch.randn(experts, d, device="cuda", generator=g).bfloat16() for _ in range(4)]
    x = torch.randn(tokens, d, device="cuda", generator=g).bfloat16()
    want = []
    for w in ws:
        want.append(R.route_topk(x, w, None, 1)[:2])
        torch.cuda.synchronize()
    got = [R.route_topk(x, ws[i % 4], None, 1)[:2] for i in range(64)]
    torch.cuda.synchronize()
    for i, (idx, w) in enumerate(got):
        assert torch.equal(idx, want[i % 4][0]) and torch.equal(w, want[i % 4][1])
