"""Outputs with more rows than the operand that they are computed from : every kernel writes zeros from a group's last row to the end of
its tile, also where the operand ends in between."""
import pytest
import torch


def test_the_launch_block_says_how_many_rows_the_outputs_have():
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    mk = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)  # noqa: E731
    index = torch.zeros(1, dtype=torch.int32)
    kw = dict(a_major=N.MAJ_K, b_major=N.MAJ_K, epi=N.EPI_BIAS_ACT, group_base=index, group_rows=index, num_groups=1)
    with N.record_launches() as rec:
        G.launch(a0=mk(100, 64), b0=mk(32, 64), n=32, k=64, b_group_rows=32, out0=mk(128, 32), out1=mk(256, 32), **kw)
        G.launch(a0=mk(100, 64), b0=mk(32, 64), n=32, k=64, b_group_rows=32, out0=mk(128, 64), ld_out=64, **kw)
        G.launch(a0=mk(128, 64), b0=mk(128, 64), n=64, kgroup=True, m_per_group=64, out0=mk(64, 64), **dict(kw, a_major=N.MAJ_MN, b_major=N.MAJ_MN, epi=N.EPI_STORE))
    got = [N.GemmLaunch.from_buffer_copy(c[1][0]).out_rows for c in rec.calls if c[0] == "ccf_gemm_launch"]
    assert got[0] == 128 and got[1] >= 128 and got[2] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [[100], [128, 1], [256, 70], [300]], ids=str)
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("grad", [False, True])
def test_rows_behind_the_operand_are_zeroed(rows, swiglu, grad):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    e, k, n, base, cur = len(rows), 192, 288, [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    held = base[-1] + rows[-1]            # the operand ends with the last group's last row, the outputs with its tile
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, w, wg, bias = mk(held, k), mk(e, k, n) if grad else mk(e, n, k), mk(e, n, k), mk(e, n)
    pre, up = mk(cur, n), mk(cur, n)
    gb, gr = torch.tensor(base, dtype=torch.int32, device="cuda"), torch.tensor(rows, dtype=torch.int32, device="cuda")
    got = []
    for two_cta in (False, True):
        out = [torch.full((cur, n), 7.0, device="cuda").bfloat16() for _ in range(3)]
        if grad:
            kw = dict(b0=w.view(e * k, n), b_major=N.MAJ_MN, b_group_rows=k, aux0=pre, epi=N.EPI_DSWIGLU if swiglu else N.EPI_DACT,
                      **(dict(aux1=up, out1=out[1]) if swiglu else dict(act=N.ACT_GELU)))
        else:
            kw = dict(b0=w.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, bias0=bias, out1=out[1],
                      **(dict(epi=N.EPI_SWIGLU, b1=wg.view(e * n, k), bias1=bias, out2=out[2]) if swiglu
                         else dict(epi=N.EPI_BIAS_ACT, act=N.ACT_GELU)))
        G.launch(a0=x, a_major=N.MAJ_K, n=n, k=k, out0=out[0], group_base=gb, group_rows=gr, num_groups=e, two_cta=two_cta, **kw)
        G.Workspace.get("cuda").check("longer outputs")
        got.append(out[:1 + (swiglu or not grad) + (swiglu and not grad)])
    for a, b in zip(*got):
        for s, r in zip(base, rows):
            assert (a[s + r:s + (r + 127) // 128 * 128] == 0).all() and (b[s + r:s + (r + 127) // 128 * 128] == 0).all()
            assert torch.equal(a[s:s + r], b[s:s + r])
