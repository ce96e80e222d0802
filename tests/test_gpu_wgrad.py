"""Weight gradients of few rows per group (csrc/gemm_wgrad.cu) against fp32 torch references (needs a B200): fp32 sums of at most 1100
products of 8- or 11-bit mantissas, rounded once; four half units in the last place of the largest value."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.bfloat16: 4 * 2.0 ** -9, torch.float16: 4 * 2.0 ** -12}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sgd", [False, True])
@pytest.mark.parametrize("m,n", [(256, 64), (256, 96), (512, 256), (768, 1120), (2048, 2048)])   # chunk and tile edges; many tiles per pair
@pytest.mark.parametrize("rows", [[1, 0, 64, 65], [256, 255, 300, 17, 0, 1100], [190] * 12], ids=lambda r: "-".join(map(str, r[:4])))
def test_few_row_weight_gradient(rows, m, n, sgd, dtype):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)  # noqa: E731
    e, base, cur = len(rows), [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    gb, gr = torch.tensor(base, dtype=torch.int32, device="cuda"), torch.tensor(rows, dtype=torch.int32, device="cuda")
    a, b, w = mk(max(cur, 128), m), mk(max(cur, 128), n), mk(e, m, n)
    for s, r in zip(base, rows):      # rows up to the next multiple of 64 take part in the reduction: zero in one operand
        a[s + r:s + (r + 127) // 128 * 128] = 0
    out, lr, wd = w.clone(), 0.05, 0.1
    for rep in range(2):
        start = out.clone()
        G.launch(a0=a, b0=b, a_major=N.MAJ_MN, b_major=N.MAJ_MN, epi=N.EPI_STORE, n=n, kgroup=True, m_per_group=m, group_base=gb,
                 group_rows=gr, num_groups=e, out0=out, ld_out=n, few_rows=True, sgd=(lr, wd) if sgd else None)
        G.Workspace.get("cuda").check("few-row weight gradient")
        for i, (s, r) in enumerate(zip(base, rows)):
            want = a[s:s + r].float().t() @ b[s:s + r].float()
            if sgd:
                want = start[i].float() - lr * (want + wd * start[i].float())
            assert float((out[i].float() - want).abs().max()) <= TOL[dtype] * max(1e-6, float(want.abs().max()))
