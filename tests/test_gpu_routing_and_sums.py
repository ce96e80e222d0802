"""Column sums at the edges of their blocks and clusters, against fp64 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
