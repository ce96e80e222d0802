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


# groups of one popular expert and small ones: only tiles with the rows for it are cut
@pytest.mark.parametrize("rows", [[256, 40, 17], [320, 64, 193, 129], [300, 20, 17, 9], [257] * 5, [128], [192] * 37, [130] * 75],
                         ids=lambda r: f"{r[0]}x{len(r)}")
@pytest.mark.parametrize("kind", ["swiglu", "dswiglu", "combine", "combine_two"])
def test_pieces_of_rows_in_the_other_epilogues(rows, kind):
    """SwiGLU and its derivative, and rows that go back to their source (with gate weights; with a second product on top)."""
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    e, k, n, base, cur = len(rows), 192, 544, [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    g = torch.Generator(device="cuda").manual_seed(13)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, x2, w, w2, pre, up, bias = mk(cur, k), mk(cur, k), mk(e, n, k), mk(e, n, k), mk(cur, n), mk(cur, n), mk(e, n)
    gb, gr = torch.tensor(base, dtype=torch.int32, device="cuda"), torch.tensor(rows, dtype=torch.int32, device="cuda")
    slots = sum(rows)
    src = torch.full((cur,), -1, dtype=torch.int32, device="cuda")
    perm, at = torch.randperm(slots, device="cuda", generator=g).int(), 0
    for s, r in zip(base, rows):
        src[s:s + r] = perm[at:at + r]
        at += r
    gate = torch.rand(cur, device="cuda", generator=g)
    got = []
    for few in (True, False):
        out = [torch.full((cur, n), 7.0, device="cuda").bfloat16() for _ in range(3)]
        comb, done = torch.full((slots, n), 7.0, device="cuda").bfloat16(), torch.zeros(8, dtype=torch.int32, device="cuda")
        back = dict(epi=N.EPI_COMBINE, row_src=src, peer_comb=[comb.data_ptr()], peer_done=[done.data_ptr()], world=1, send_finish=1,
                    max_slots=slots, ld_out=n)
        kw = {"swiglu": dict(epi=N.EPI_SWIGLU, b0=w.view(e * n, k), b1=w2.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, bias0=bias,
                             bias1=bias, out0=out[0], out1=out[1], out2=out[2]),
              "dswiglu": dict(epi=N.EPI_DSWIGLU, b0=w.view(e * k, n), b_major=N.MAJ_MN, b_group_rows=k, aux0=pre, aux1=up, out0=out[0],
                              out1=out[1]),
              "combine": dict(b0=w.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, bias0=bias, row_gate=gate, **back),
              "combine_two": dict(a1=x2, b0=w.view(e * k, n), b1=w2.view(e * k, n), b_major=N.MAJ_MN, b_group_rows=k, kseg=2, **back)}[kind]
        G.launch(a0=x, a_major=N.MAJ_K, n=n, k=k, group_base=gb, group_rows=gr, num_groups=e, few_rows=few, two_cta=not few, **kw)
        G.Workspace.get("cuda").check("pieces")
        got.append(out + [comb, done])
    for i, (a, b) in enumerate(zip(*got)):
        if i < 3:
            for s, r in zip(base, rows):
                up_to = s + (r + 63) // 64 * 64
                assert torch.equal(a[s:up_to], b[s:up_to])
                if kind != "combine" and kind != "combine_two" and i < (3 if kind == "swiglu" else 2):
                    assert (a[s + r:up_to] == 0).all()
        else:
            assert torch.equal(a, b)
