"""The GEMM for few rows per group (csrc/gemm_swap.cu): a row's result is the same to the bit whatever is routed beside it, and the
same as on the CTA-pair kernel: both sum over k in order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

FIRST = 40
BESIDE = [[30] * 7, [250, 0, 1, 17, 128, 64, 99], [0] * 7, [300] * 7]


def _launch(rows, n, k, dtype, epi, x0, w, aux0, swap):
    """The first group's rows of one launch; the other groups get other data each time."""
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    e = len(rows)
    base = [384 * i for i in range(e)]
    gb, gr = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (base, rows))
    x = torch.randn(384 * e, k, device="cuda").to(dtype)
    x[:FIRST] = x0
    out = torch.zeros(384 * e, n, device="cuda", dtype=dtype)
    kw = dict(a0=x, a_major=N.MAJ_K, n=n, k=k, group_base=gb, group_rows=gr, num_groups=e, few_rows=swap)
    if epi == "act":
        G.launch(b0=w.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, epi=N.EPI_BIAS_ACT, out0=out, act=N.ACT_NONE, **kw)
    elif epi == "dact":
        aux = torch.randn(384 * e, n, device="cuda").to(dtype)
        aux[:FIRST] = aux0
        G.launch(b0=w.view(e * k, n), b_major=N.MAJ_MN, b_group_rows=k, epi=N.EPI_DACT, out0=out, aux0=aux, act=N.ACT_RELU, **kw)
    else:
        src = torch.full((384 * e,), -1, dtype=torch.int32, device="cuda")
        for s, r in zip(base, rows):
            src[s:s + r] = torch.arange(s, s + r, dtype=torch.int32, device="cuda")
        done = torch.zeros(8, dtype=torch.int32, device="cuda")
        G.launch(b0=w.view(e * n, k), b_major=N.MAJ_K, b_group_rows=n, epi=N.EPI_COMBINE, row_src=src, peer_comb=[out.data_ptr()],
                 peer_done=[done.data_ptr()], send_finish=1, max_slots=384 * e, ld_out=n, **kw)
    G.Workspace.get("cuda").check("rows beside each other")
    return out[:FIRST].clone()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("epi", ["act", "dact", "combine"])
@pytest.mark.parametrize("n,k", [(512, 2048), (1024, 4096), (2560, 1088)])
def test_result_of_a_row_does_not_depend_on_the_others(n, k, epi, dtype):
    torch.manual_seed(n + k)
    x0, aux0 = torch.randn(FIRST, k, device="cuda").to(dtype), torch.randn(FIRST, n, device="cuda").to(dtype)
    w = (torch.randn(8, n, k, device="cuda") * k ** -0.5).to(dtype)
    want = _launch([FIRST] + BESIDE[0], n, k, dtype, epi, x0, w, aux0, swap=False)
    for beside in BESIDE:
        assert torch.equal(_launch([FIRST] + beside, n, k, dtype, epi, x0, w, aux0, swap=True), want)
