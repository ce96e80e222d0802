"""The last round of the kernel for few rows, whose tiles come in pieces of their rows (needs a B200): the bits of the kernel on CTA
pairs, which knows no pieces, and zeros up to the next 64 rows where a reduction over rows reads the output."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 128 rows are the smallest that are cut; 300 and 320 rows come in two parts where they are whole; with 40 tiles of 74 pairs
# none is cut, with 37 they are halves; 75 tiles leave one for a second round
@pytest.mark.parametrize("rows", [[127], [128], [129, 300, 1], [320] * 3, [256, 0, 200, 17], [257] * 5, [192] * 37, [192] * 40, [130] * 75],
                         ids=lambda r: f"{r[0]}x{len(r)}")
@pytest.mark.parametrize("n", [256, 544])
@pytest.mark.parametrize("grad", [False, True])
def test_pieces_of_rows(rows, n, grad):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    e, k, base, cur = len(rows), 192, [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    g = torch.Generator(device="cuda").manual_seed(11)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, w, pre, bias = mk(cur, k), mk(e, k, n) if grad else mk(e, n, k), mk(cur, n), mk(e, n)
    gb, gr = torch.tensor(base, dtype=torch.int32, device="cuda"), torch.tensor(rows, dtype=torch.int32, device="cuda")
    got = []
    for few in (True, False):
        out, out1 = torch.full((cur, n), 7.0, device="cuda").bfloat16(), torch.full((cur, n), 7.0, device="cuda").bfloat16()
        if grad:
            kw = dict(b0=w.view(e * k, n), b_major=N.MAJ_MN, epi=N.EPI_DACT, b_group_rows=k, aux0=pre)
        else:
            kw = dict(b0=w.view(e * n, k), b_major=N.MAJ_K, epi=N.EPI_BIAS_ACT, b_group_rows=n, bias0=bias, out1=out1)
        G.launch(a0=x, a_major=N.MAJ_K, n=n, k=k, act=N.ACT_GELU, out0=out, group_base=gb, group_rows=gr, num_groups=e, few_rows=few,
                 two_cta=not few, **kw)
        G.Workspace.get("cuda").check("pieces")
        got.append((out, out1))
    for a, b in zip(*got):
        for s, r in zip(base, rows):
            up = s + (r + 63) // 64 * 64
            assert torch.equal(a[s:up], b[s:up])
            if not (grad and a is got[0][1]):
                assert (a[s + r:up] == 0).all()
