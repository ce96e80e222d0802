"""Column sums and the router's split over d at the edges of their blocks and clusters, against fp64 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,d,e,k,dtype,bias", [(1, 128, 3, 2, torch.bfloat16, True), (127, 256, 8, 2, torch.float16, False),
                                               (129, 768, 33, 4, torch.bfloat16, True), (600, 4096, 256, 8, torch.bfloat16, True),
                                               (2500, 512, 64, 2, torch.float16, True), (9473, 1024, 16, 1, torch.bfloat16, True),
                                               (300, 672, 130, 2, torch.bfloat16, False)])
def test_router_splits(t, d, e, k, dtype, bias):
    """One, two, four and eight CTAs per row tile, ragged rows and columns: logits against fp64 (the operands are exact in
    fp32 and the sums are fp32: an error of a few 2^-24 of the sum of magnitudes), selection from exactly those logits."""
    from ccfuser_b200.gates import topk_softmax_reference
    from ccfuser_b200.ops.gemm import Workspace
    from ccfuser_b200.ops.router import fused_router
    torch.manual_seed(t)
    x = torch.randn(t, d, device="cuda").to(dtype)
    w = (torch.randn(e, d, device="cuda") * 0.05).to(dtype)
    b = (torch.randn(e, device="cuda") * 0.1).to(dtype) if bias else None
    with torch.no_grad():
        idx, wt, logits = fused_router(x, w, b, k, want_logits=True)
    Workspace.get(x.device).check("router")
    ref = x.double() @ w.double().t() + (b.double() if bias else 0)
    scale = x.double().abs() @ w.double().abs().t() + 1
    assert ((logits.double() - ref).abs() <= scale * 2.0 ** -18).all()
    ridx, rw = topk_softmax_reference(logits, k)
    assert torch.equal(idx.long(), ridx) and torch.allclose(wt, rw, atol=1e-6)


@pytest.mark.parametrize("rows,n,fp16", [([4000, 130, 0, 5000], 1024, False), ([1] * 3, 8, True), ([63, 64, 65, 129] * 16, 256, False),
                                        ([700], 136, True), ([300] * 64, 2048, False)])
def test_column_sums_shared_by_a_cluster(rows, n, fp16):
    """One to eight blocks per (column block, group); fp32 sums (2^-24 of the sum of magnitudes per addition chain of at
    most a few hundred), one rounding, the same bits every time."""
    from ccfuser_b200 import native as N
    dt = torch.float16 if fp16 else torch.bfloat16
    base, acc = [], 0
    for r in rows:
        base.append(acc)
        acc += (r + 127) // 128 * 128
    x = torch.randn(max(acc, 128), n, device="cuda").to(dt)
    gb = torch.tensor(base, dtype=torch.int32, device="cuda")
    gr = torch.tensor(rows, dtype=torch.int32, device="cuda")
    outs = []
    for _ in range(2):
        out = torch.empty(len(rows), n, dtype=dt, device="cuda")
        N.check(N.load().ccf_colsum_grouped(x.data_ptr(), n, n, len(rows), gb.data_ptr(), gr.data_ptr(), out.data_ptr(),
                                            int(fp16), N.stream_ptr()), "ccf_colsum_grouped")
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    ref = torch.stack([x[b:b + r].double().sum(0) for b, r in zip(base, rows)])
    mag = torch.stack([x[b:b + r].double().abs().sum(0) for b, r in zip(base, rows)])
    ulp = 2.0 ** (-11 if fp16 else -8)
    assert ((outs[0].double() - ref).abs() <= ref.abs() * ulp + mag * 2.0 ** -16 + 1e-7).all()
