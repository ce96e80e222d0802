"""Grouped GEMM with the weights on the M side (csrc/gemm_swap.cu) against fp32 torch references (needs a B200). Inputs carry 8 or 11
bits of mantissa, sums are fp32, results are rounded once: 2^-8 (bf16) or 2^-11 (fp16) of a value, and the activation's fp32
polynomial is far below that; the bound is four half units in the last place of the largest value."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

TOL = {torch.bfloat16: 4 * 2.0 ** -9, torch.float16: 4 * 2.0 ** -12}

# rows per group at the edges of boxes (16), chunks (32), parts (160), tiles (256, 320) and beyond; with few tiles for 74 CTA pairs
# their k-blocks are shared, with many only the last ones' are, and every accumulator is used several times
ROWS = [[2, 0, 1, 16, 17], [33, 128, 0, 160], [161, 256, 255], [257, 5, 320, 321], [700, 64, 129], [3] * 40, [272, 250] * 8]
SHAPES = [(64, 96), (256, 1024), (640, 576), (1024, 4096), (4096, 96)]    # n, k


def _data(rows, n, k, dtype, seed):
    from ccfuser_b200.ops import gemm as G
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s, std=1.0: (torch.randn(*s, device="cuda", generator=g) * std).to(dtype)  # noqa: E731
    base, cur = [], 0
    for r in rows:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    gb = torch.tensor(base, dtype=torch.int32, device="cuda")
    gr = torch.tensor(rows, dtype=torch.int32, device="cuda")
    return G, mk, base, gb, gr, max(cur, 128)


def _check(got, ref, rows, base, dtype, zeros):
    tol = TOL[dtype] * max(float(r.abs().max()) for r in ref if r.numel())
    for s, r, want in zip(base, rows, ref):
        assert float((got[s:s + r].float() - want).abs().max()) <= tol if r else True
        if r and zeros:
            assert (got[s + r:s + (r + 63) // 64 * 64] == 0).all()
            assert (got[s + (r + 63) // 64 * 64:s + (r + 127) // 128 * 128] == 7).all()
        elif r:
            assert (got[s + r:s + (r + 127) // 128 * 128] == 7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("rows", ROWS, ids=lambda r: "-".join(map(str, r[:5])))
def test_swapped_kernel(rows, n, k, dtype):
    from ccfuser_b200 import native as N
    G, mk, base, gb, gr, total = _data(rows, n, k, dtype, 11)
    e, out = len(rows), lambda: torch.full((total, n), 7.0, device="cuda", dtype=dtype)  # noqa: E731
    x, x2 = mk(total, k), mk(total, k)
    for s, r in zip(base, rows):      # what lies behind a group's rows is never looked at
        x[s + r:s + (r + 127) // 128 * 128] = float("nan")
    w, wg = mk(e, n, k, std=k ** -0.5), mk(e, n, k, std=k ** -0.5)
    wt, wgt = w.transpose(1, 2).contiguous(), wg.transpose(1, 2).contiguous()    # [e, k, n]
    b, bg = mk(e, n), mk(e, n)
    part = lambda t: [t[s:s + r].float() for s, r in zip(base, rows)]  # noqa: E731
    lin = lambda xs, ws: [p @ v.float().t() for p, v in zip(xs, ws)]  # noqa: E731
    common = dict(a_major=N.MAJ_K, n=n, k=k, group_base=gb, group_rows=gr, num_groups=e, few_rows=True)
    fwd = dict(a0=x, b0=w.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, **common)
    bwd = dict(a0=x, b0=wt.view(e * k, n), b_major=N.MAJ_MN, b_group_rows=k, **common)
    ws = G.Workspace.get("cuda")
    plain = lin(part(x), w)
    for rep in range(2):     # a second launch finds the counters of shared sums as the first did
        pre, h, h1 = out(), out(), out()
        G.launch(epi=N.EPI_BIAS_ACT, out0=h, out1=pre, bias0=b, act=N.ACT_GELU, **fwd)
        G.launch(epi=N.EPI_BIAS_ACT, out0=h1, act=N.ACT_NONE, **fwd)
        z = [p + v.float() for p, v in zip(plain, b)]
        _check(pre, z, rows, base, dtype, True)
        _check(h, [F.gelu(v) for v in z], rows, base, dtype, True)
        _check(h1, plain, rows, base, dtype, False)
        gp, up, y = out(), out(), out()
        G.launch(epi=N.EPI_SWIGLU, b1=wg.view(e * n, k), out0=y, out1=gp, out2=up, bias0=b, bias1=bg, **fwd)
        zg = [p + v.float() for p, v in zip(lin(part(x), wg), bg)]
        _check(gp, zg, rows, base, dtype, True)
        _check(up, z, rows, base, dtype, True)
        _check(y, [F.silu(p) * q for p, q in zip(zg, z)], rows, base, dtype, True)
        # backward: the same products with weights [k, n]
        aux, aux2, d0, d1 = mk(total, n), mk(total, n), out(), out()
        G.launch(epi=N.EPI_DACT, out0=d0, aux0=aux, act=N.ACT_GELU, **bwd)
        ref = []
        for p, v in zip(plain, part(aux)):
            v.requires_grad_(True)
            ref.append(p * torch.autograd.grad(F.gelu(v).sum(), v)[0])
        _check(d0, ref, rows, base, dtype, True)
        d0 = out()
        G.launch(epi=N.EPI_DSWIGLU, out0=d0, out1=d1, aux0=aux, aux1=aux2, **bwd)
        sg = [torch.sigmoid(v) for v in part(aux)]
        _check(d0, [p * u * s * (1 + v * (1 - s)) for p, u, s, v in zip(plain, part(aux2), sg, part(aux))], rows, base, dtype, True)
        _check(d1, [p * v * s for p, s, v in zip(plain, sg, part(aux))], rows, base, dtype, True)
        # combine: rows scattered to slots; two segments of k
        slots = sum(rows)
        perm = torch.randperm(slots, device="cuda").int()
        src, gate = torch.full((total,), -1, dtype=torch.int32, device="cuda"), torch.zeros(total, device="cuda")
        cur = 0
        for s, r in zip(base, rows):
            src[s:s + r], gate[s:s + r] = perm[cur:cur + r], torch.rand(r, device="cuda") + 0.1
            cur += r
        for mode in (fwd, dict(bwd, a1=x2, b1=wgt.view(e * k, n), kseg=2)):
            comb = torch.full((slots + 1, n), 7.0, device="cuda", dtype=dtype)
            done = torch.zeros(8, dtype=torch.int32, device="cuda")
            scale = gate if mode is fwd else None
            G.launch(epi=N.EPI_COMBINE, row_src=src, row_gate=scale, peer_comb=[comb.data_ptr()], peer_done=[done.data_ptr()], world=1,
                     send_finish=1, max_slots=slots, bias0=b if mode is fwd else None, ld_out=n, **mode)
            want = [(p + v.float()) for p, v in zip(plain, b)] if mode is fwd else [p + q for p, q in zip(plain, lin(part(x2), wg))]
            top = max(float(v.abs().max()) for v in want if v.numel())
            for s, r, v in zip(base, rows, want):
                if r:
                    v = v * gate[s:s + r, None] if mode is fwd else v
                    assert float((comb[src[s:s + r].long()].float() - v).abs().max()) <= TOL[dtype] * 1.1 * top
            assert (comb[slots] == 7).all() and int(done[0]) == slots * G.combine_units(n, few_rows=True) + 1
    ws.check("swapped kernel")
