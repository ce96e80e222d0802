"""Completion counts of the GEMM + combine launch: every kernel and tile width reports n / 32 per row to the rank the row came from."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [dict(two_cta=True), dict(two_cta=False), dict(two_cta=False, bn=128), dict(few_rows=True)],
                         ids=["pair", "one_cta", "one_cta_128", "few_rows"])
@pytest.mark.parametrize("n", [64, 96, 256, 320, 1056])
def test_every_kernel_counts_the_same(n, kernel):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    torch.manual_seed(n)
    k, rows = 192, [0, 1, 127, 130, 300]
    base, cur = [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    x = torch.randn(cur, k, device="cuda").bfloat16()
    w = (torch.randn(len(rows), n, k, device="cuda") * k ** -0.5).bfloat16()
    src = torch.full((cur,), -1, dtype=torch.int32)
    slot = [0, 0]
    for b, r in zip(base, rows):
        for i in range(r):                   # rows of two ranks in turn; both ranks' buffers are on this GPU
            rank = (b + i) % 3 % 2
            src[b + i] = rank << 24 | slot[rank]
            slot[rank] += 1
    comb = [torch.zeros(max(slot), n, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    done = torch.zeros(2, dtype=torch.int32, device="cuda")
    gb, gr = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (base, rows))
    G.launch(a0=x, b0=w.view(-1, k), a_major=N.MAJ_K, b_major=N.MAJ_K, epi=N.EPI_COMBINE, n=n, k=k, group_base=gb, group_rows=gr,
             num_groups=len(rows), b_group_rows=n, row_src=src.cuda(), peer_comb=[c.data_ptr() for c in comb],
             peer_done=[done.data_ptr(), done.data_ptr() + 4], world=2, send_finish=1, max_slots=max(slot), ld_out=n, **kernel)
    G.Workspace.get("cuda").check("combine units")
    assert done.tolist() == [s * G.combine_units(n) + 1 for s in slot] == [s * (n // 32) + 1 for s in slot]
    for b, r, v in zip(base, rows, w):
        if r:
            want = x[b:b + r].float() @ v.float().t()
            for rank in range(2):
                sel = (src[b:b + r] >> 24) == rank
                got = comb[rank][(src[b:b + r][sel] & 0xffffff).long().cuda()].float()
                # bf16 inputs, fp32 sums of 192 terms, one rounding of the result: four half units of the largest value
                assert float((got - want[sel.cuda()]).abs().max()) <= 4 * 2.0 ** -9 * float(want.abs().max()) if sel.any() else True
