"""Arrival gating of the GEMM for few rows per group (csrc/gemm_swap.cu): tiles wait for the counters of the 128-row tiles that
their rows lie in, here set by the test. A wait that nothing ends gives up within its limit and says where."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# row tiles of 240 rows over three counters (700), of 320 over three (320), of one row, none
ROWS = [700, 0, 1, 320, 128, 129]
N_, K = 512, 320


def _setup():
    torch.manual_seed(1)
    base, cur = [], 0
    for r in ROWS:
        base.append(cur)
        cur += (r + 127) // 128 * 128
    flags = torch.zeros(cur // 128 + 1, dtype=torch.int32)
    for b, r in zip(base, ROWS):
        for t in range((r + 127) // 128):
            flags[b // 128 + t] = min(128, r - 128 * t)
    x = torch.randn(cur, K, device="cuda").bfloat16()
    w = (torch.randn(len(ROWS), N_, K, device="cuda") * K ** -0.5).bfloat16()
    return base, cur, flags, x, w


def _launch(base, total, flags, x, w, total_index, **kw):
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    out = torch.full((total, N_), 7.0, device="cuda", dtype=torch.bfloat16)
    gb, gr = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (base, ROWS))
    G.launch(a0=x, b0=w.view(-1, K), a_major=N.MAJ_K, b_major=N.MAJ_K, epi=N.EPI_BIAS_ACT, n=N_, k=K, group_base=gb, group_rows=gr,
             num_groups=len(ROWS), b_group_rows=N_, out0=out, act=N.ACT_NONE, tile_flags=flags, total_index=total_index, few_rows=True, **kw)
    torch.cuda.synchronize()
    return out


def _check(out, base, x, w):
    for b, r, v in zip(base, ROWS, w):
        if r:
            # bf16 inputs, fp32 sums of 320 terms, one rounding of the result: four half units of the largest value
            want = x[b:b + r].float() @ v.float().t()
            assert float((out[b:b + r].float() - want).abs().max()) <= 4 * 2.0 ** -9 * float(want.abs().max())


@pytest.mark.parametrize("counted", ["every tile", "the total", "the total behind"])
def test_tiles_whose_rows_are_there(counted):
    """The count of all rows lets later tiles pass without a look at their own; behind it every tile looks."""
    from ccfuser_b200.ops import gemm as G
    base, total, flags, x, w = _setup()
    index = -1 if counted == "every tile" else flags.numel() - 1
    flags[-1] = sum(ROWS) - (counted == "the total behind")
    _check(_launch(base, total, flags.cuda(), x, w, index), base, x, w)
    G.Workspace.get("cuda").check("gated tiles")


@pytest.mark.parametrize("tile", [2, 5, 6, 8])      # third and last counter of the 700 rows, the one row, the 320
def test_a_row_that_never_comes(tile):
    from ccfuser_b200.errors import MoECommTimeout
    from ccfuser_b200.ops import gemm as G
    base, total, flags, x, w = _setup()
    ws = G.Workspace.get("cuda")
    short = flags.clone()
    short[tile] -= 1
    short[-1] = sum(ROWS) - 1
    _launch(base, total, short.cuda(), x, w, flags.numel() - 1, wait_ns=20_000_000)
    with pytest.raises(MoECommTimeout):
        ws.check("gated tiles")
    # the next launch finds nothing of the one that was given up
    assert not ws.sched.any()
    flags[-1] = sum(ROWS)
    _check(_launch(base, total, flags.cuda(), x, w, flags.numel() - 1), base, x, w)
    ws.check("gated tiles")


# the completion counters wrap around: what counts is how far the counter is from its target
@pytest.mark.parametrize("count,target,reached", [(-(1 << 31) + 4, (1 << 31) - 8, True), ((1 << 31) - 8, -(1 << 31) + 4, False),
                                                  (-3, -3, True), (5, 6, False), (2, -2, True)])
def test_a_counter_that_has_wrapped_around(count, target, reached):
    from ccfuser_b200 import native as N
    flag = torch.tensor([count], dtype=torch.int32, device="cuda")
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    N.check(N.load().ccf_wait_probe(flag.data_ptr(), target, 5_000_000, status.data_ptr(), N.stream_ptr()), "probe")
    torch.cuda.synchronize()
    assert (int(status[0]) == 0) == reached
