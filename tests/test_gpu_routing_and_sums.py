"""Routing + plan in one kernel, slot reduction, router weight gradient, column sums and the router's split over d: at the
edges of their blocks, clusters and dispatch rules, against fp64 sums or the separate kernels they replace."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan_args(N, e, kept, max_rows, epoch):
    i32 = dict(dtype=torch.int32, device="cuda")
    out = {k: torch.full((e,), -7, **i32) for k in ("dst_base", "group_base", "group_rows", "local_begin", "local_rows")}
    out["sent_rows"], out["table_copy"] = torch.full((8,), -7, **i32), torch.full((e,), -7, **i32)
    keep = {"table": torch.zeros(e, **i32), "flag": torch.zeros(8, **i32), "status": torch.zeros(2, **i32)}
    p = N.PlanArgs()
    p.count_kept = kept.data_ptr()
    p.peer_table[0], p.peer_flag[0] = keep["table"].data_ptr(), keep["flag"].data_ptr()
    for k, t in out.items():
        setattr(p, k, t.data_ptr())
    p.status, p.wait_limit_ns = keep["status"].data_ptr(), 1_000_000_000
    p.world, p.my_rank, p.e_total, p.e_loc, p.epoch, p.max_rows = 1, 0, e, e, epoch, max_rows
    return p, out, keep


@pytest.mark.parametrize("slots,e,cap,first", [(1, 1, 1, 0), (31, 4, 100, 2), (1024, 64, 20, 0), (1025, 256, 1 << 20, 255),
                                              (4097, 64, 50, 3), (16384, 8, 2000, 0), (32768, 64, 1 << 20, 0),
                                              (40000, 16, 2600, 5), (65536, 256, 300, 128)])
def test_route_plan_equals_the_separate_kernels(slots, e, cap, first):
    """Every output of the one-kernel form is the one of ccf_route_ordered + ccf_plan, with a receive buffer that some rows
    do not fit and ids outside the table; raw_order lists all routed slots by expert in slot order."""
    from ccfuser_b200 import native as N
    lib = N.load()
    g = torch.Generator(device="cuda").manual_seed(slots)
    expert = torch.randint(-1, e + 1, (slots,), dtype=torch.int32, device="cuda", generator=g)   # -1 and e: not routed
    i32 = dict(dtype=torch.int32, device="cuda")
    nb = (slots + 1023) // 1024
    max_rows = max(128, slots // 2 // 128 * 128)
    res = []
    for one in (False, True):
        t = {"pos": torch.zeros(slots, **i32), "raw": torch.zeros(e, **i32), "kept": torch.zeros(e, **i32),
             "order_off": torch.zeros(e + 1, **i32), "sorted_slot": torch.full((slots,), -1, **i32),
             "slot_row": torch.zeros(slots, **i32)}
        p, out, keep = _plan_args(N, e, t["kept"], max_rows, 3)
        if one:
            raw_order = torch.full((N.MAX_GROUPS + slots,), -1, **i32)
            N.check(lib.ccf_route_plan(expert.data_ptr(), slots, e, cap, t["pos"].data_ptr(), t["raw"].data_ptr(),
                                       t["kept"].data_ptr(), t["order_off"].data_ptr(), t["sorted_slot"].data_ptr(),
                                       t["slot_row"].data_ptr(), first, raw_order.data_ptr(), C.byref(p), None,
                                       N.stream_ptr()), "ccf_route_plan")
        else:
            bh, bo, ticket = torch.zeros(nb * e, **i32), torch.zeros(nb * e, **i32), torch.zeros(1, **i32)
            N.check(lib.ccf_route_ordered(expert.data_ptr(), slots, e, cap, t["pos"].data_ptr(), bh.data_ptr(), bo.data_ptr(),
                                          t["raw"].data_ptr(), t["kept"].data_ptr(), ticket.data_ptr(),
                                          t["order_off"].data_ptr(), t["sorted_slot"].data_ptr(), t["slot_row"].data_ptr(),
                                          first, N.stream_ptr()), "ccf_route_ordered")
            N.check(lib.ccf_plan(C.byref(p), N.stream_ptr()), "ccf_plan")
        torch.cuda.synchronize()
        res.append({**t, **out, "status": keep["status"]})
    for k in res[0]:
        assert torch.equal(res[0][k], res[1][k]), k
    # the layout itself, from the counts
    kept = res[1]["kept"].cpu()
    padded = (kept + 127) // 128 * 128
    base = torch.cumsum(padded, 0) - padded
    assert torch.equal(res[1]["group_base"].cpu().long(), base)
    assert int(res[1]["sent_rows"][0]) == int(torch.minimum(kept, (max_rows - base).clamp(min=0)).sum())
    ids = expert.cpu()
    for k in range(e):
        ex = (first + k) % e
        want = (ids == ex).nonzero().flatten().int()
        start = int(raw_order[ex])
        assert torch.equal(raw_order[N.MAX_GROUPS + start:N.MAX_GROUPS + start + want.numel()].cpu(), want)


def test_route_plan_leaves_other_sizes_to_the_separate_kernels():
    from ccfuser_b200 import native as N
    kept = torch.zeros(4, dtype=torch.int32, device="cuda")
    p, _, _ = _plan_args(N, 4, kept, 128, 1)
    for slots in (0, N.ROUTE_CLUSTER_SLOTS + 1):
        assert N.load().ccf_route_plan(0, slots, 4, 1, 0, 0, 0, 0, 0, 0, 0, 0, C.byref(p), None, N.stream_ptr()) == 1


@pytest.mark.parametrize("tokens,k,d,fp16", [(1, 1, 64, False), (129, 2, 768, True), (77, 3, 4096, False), (33, 8, 512, True),
                                            (40, 9, 256, False), (65, 2, 8192, False)])
def test_combine_reduce(tokens, k, d, fp16):
    from ccfuser_b200 import native as N
    dt = torch.float16 if fp16 else torch.bfloat16
    torch.manual_seed(tokens)
    comb = torch.randn(tokens * k, d, device="cuda").to(dt)
    row = torch.randint(-1, 5, (tokens * k,), dtype=torch.int32, device="cuda")
    comb[row < 0] = float("nan")                                     # rows of dropped slots are never read
    y = torch.empty(tokens, d, dtype=dt, device="cuda")
    N.check(N.load().ccf_combine_reduce(comb.data_ptr(), row.data_ptr(), y.data_ptr(), tokens, k, d, int(fp16),
                                        N.stream_ptr()), "ccf_combine_reduce")
    ref = torch.where((row >= 0).unsqueeze(1), comb.double(), torch.zeros((), dtype=torch.float64, device="cuda"))
    ref = ref.view(tokens, k, d).sum(1)
    # one rounding to the element type after fp32 sums: with 8 (bf16) or 11 (fp16) significant bits half a unit in the last
    # place is at most 2^-8 or 2^-11 of the value
    ulp = 2.0 ** (-11 if fp16 else -8)
    assert ((y.double() - ref).abs() <= ref.abs() * ulp * 1.01 + 1e-6).all()


@pytest.mark.parametrize("act,e,k,t,cf,dtype", [("gelu", 4, 2, 300, None, torch.bfloat16), ("relu", 16, 1, 129, 1.0, torch.float16),
                                               ("swiglu", 8, 3, 1000, 0.5, torch.bfloat16),
                                               ("gelu", 64, 2, 4500, 1.25, torch.bfloat16), ("gelu", 2, 2, 1, None, torch.float16)])
def test_one_node_layer_equals_router_then_experts(act, e, k, t, cf, dtype):
    """Router and experts as one autograd node against the two nodes (same kernels for everything but the router's
    backward): outputs are the same bits, dx differs by roundings of its two addends, the router's gradients by the
    rounding of the dense logit gradient the two-node form multiplies with."""
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(e + t)
    d, f = 256, 512
    cfg = MoEConfig(d_model=d, d_ffn=f, num_experts=e, top_k=k, capacity_factor=cf, activation=act, dtype=dtype,
                    backend="fused", max_tokens=t)
    layer = MoELayer(cfg, device="cuda")
    fm = layer._fused_impl()
    x = torch.randn(t, d, device="cuda", dtype=dtype).requires_grad_()
    gy = torch.randn(t, d, device="cuda", dtype=dtype)
    got = []
    for one in (False, True):
        assert fm.one_node(x)
        for p in [x, *layer.parameters()]:
            p.grad = None
        y = layer(x) if one else fm.run_experts(x, *fm.route(x))
        y.backward(gy)
        got.append({"y": y.detach(), "x": x.grad, **{n: p.grad for n, p in layer.named_parameters()}})
    layer.check_status()
    eps = 2.0 ** (-10 if dtype == torch.float16 else -7)
    for n in got[0]:
        a, b = got[0][n].double(), got[1][n].double()
        if n.startswith("experts") or n == "y":
            assert torch.equal(a, b), n
        else:
            assert (a - b).norm() <= 2 * eps * a.norm() + 1e-6, n
    layer.release()


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


@pytest.mark.parametrize("two_cta", [False, True])
@pytest.mark.parametrize("groups", [1, 31, 33, 64, 256])
def test_tile_tables_of_many_groups(groups, two_cta):
    """The warp-parallel tile tables of both GEMM kernels: ragged and empty groups across the 32-group scan steps."""
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    g = torch.Generator().manual_seed(groups)
    rows = torch.randint(0, 300, (groups,), generator=g)
    rows[torch.randint(0, groups, (groups // 3,), generator=g)] = 0
    rows[-1] = 129
    padded = (rows + 127) // 128 * 128
    base = torch.cumsum(padded, 0) - padded
    total = int(padded.sum()) + 128
    k, n = 64, 256
    x = torch.randn(total, k, device="cuda").bfloat16()
    w = (torch.randn(groups * n, k, device="cuda") * 0.1).bfloat16()
    out = torch.zeros(total, n, dtype=torch.bfloat16, device="cuda")
    gb, gr = base.int().cuda(), rows.int().cuda()
    ws = G.launch(a0=x, b0=w, a_major=N.MAJ_K, b_major=N.MAJ_K, epi=N.EPI_STORE, n=n, k=k, group_base=gb, group_rows=gr,
                  num_groups=groups, b_group_rows=n, out0=out, two_cta=two_cta)
    ws.check("tables")
    for i in range(groups):
        b, r = int(base[i]), int(rows[i])
        ref = x[b:b + r].double() @ w[i * n:(i + 1) * n].double().t()
        assert ((out[b:b + r].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4).all(), i


@pytest.mark.parametrize("a_rows,bn,two_cta,rows", [(32, 128, False, [1, 32, 0, 31, 7]), (32, 256, False, [32, 2]), (64, 128, False, [64, 33, 1]),
                                                    (64, 256, False, [63, 0, 64]), (0, 128, False, [128, 97, 1, 65]),
                                                    (0, 256, False, [33, 130, 300, 96]), (0, 256, True, [1, 129, 160, 257, 300, 512])])
@pytest.mark.parametrize("k", [64, 1024])
def test_row_bound(a_rows, bn, two_cta, rows, k):
    """Pipeline geometries of the one-CTA kernel (rows of A per stage x tile width) and the CTA-pair kernel at ragged rows:
    what the stages hold beyond a tile's rows must not reach a stored row. The rows of A outside the groups hold NaN."""
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    torch.manual_seed(k + len(rows))
    base, acc = [], 0
    for r in rows:
        base.append(acc)
        acc += (r + 127) // 128 * 128
    n, groups = 384, len(rows)
    x = torch.full((max(acc, 128) + 128, k), float("nan"), device="cuda", dtype=torch.bfloat16)
    for b, r in zip(base, rows):
        x[b:b + r] = torch.randn(r, k, device="cuda").bfloat16()
    w = (torch.randn(groups * n, k, device="cuda") * 0.1).bfloat16()
    out = torch.full((x.shape[0], n), 7.0, dtype=torch.bfloat16, device="cuda")
    ws = G.launch(a0=x, b0=w, a_major=N.MAJ_K, b_major=N.MAJ_K, epi=N.EPI_STORE, n=n, k=k,
                  group_base=torch.tensor(base, dtype=torch.int32, device="cuda"),
                  group_rows=torch.tensor(rows, dtype=torch.int32, device="cuda"), num_groups=groups, b_group_rows=n, out0=out,
                  two_cta=two_cta, bn=bn, a_rows=a_rows)
    ws.check("row bound")
    for i, (b, r) in enumerate(zip(base, rows)):
        ref = x[b:b + r].double() @ w[i * n:(i + 1) * n].double().t()
        # bf16 result of fp32 sums of k products of order 0.1
        assert ((out[b:b + r].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4).all(), i
        assert (out[b + r:b + (r + 127) // 128 * 128] == 7.0).all()


def test_row_bound_is_refused_where_it_does_not_exist():
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    x = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16)
    gb, gr = G.single_group(32, "cuda")
    for kw in (dict(two_cta=True, a_rows=32), dict(two_cta=False, a_rows=48), dict(two_cta=False, a_rows=32, a_major=N.MAJ_MN)):
        kw = {"a_major": N.MAJ_K, **kw}
        with pytest.raises(RuntimeError):
            G.launch(a0=x, b0=x, b_major=N.MAJ_K, epi=N.EPI_STORE, n=128, k=64, group_base=gb, group_rows=gr, num_groups=1,
                     b_group_rows=128, out0=x, **kw)


@pytest.mark.parametrize("t,e,k,act", [(1, 16, 2, "gelu"), (16, 16, 2, "swiglu"), (40, 4, 1, "relu"), (64, 8, 1, "gelu"), (33, 64, 2, "gelu")])
def test_few_token_layer_uses_the_bound_and_matches_the_oracle(t, e, k, act):
    """Training and inference calls around the bounds of the small pipeline geometries, against the fp32 oracle on the same
    routing decisions."""
    from ccfuser_b200 import MoEConfig, MoELayer
    from ccfuser_b200.ops.reference import dense_moe_oracle
    torch.manual_seed(t * e)
    cfg = MoEConfig(d_model=256, d_ffn=512, num_experts=e, top_k=k, activation=act, dtype=torch.bfloat16, backend="fused",
                    max_tokens=128)
    layer = MoELayer(cfg, device="cuda")
    x = torch.randn(t, 256, device="cuda", dtype=torch.bfloat16).requires_grad_()
    fm = layer._fused_impl()
    y = layer(x)
    gy = torch.randn_like(y)
    y.backward(gy)
    layer.check_status()
    with torch.no_grad():
        assert torch.equal(layer(x.detach()), y)           # inference form: same kernels without the pre-activations
        idx, w = fm.route(x.detach())
    params = {n.replace("experts.", "").replace("gate.gate.", "gate."): p.detach().float().requires_grad_() for n, p in layer.named_parameters()}
    xf = x.detach().float().requires_grad_()
    sc = w.detach().clone()
    (ref,) = dense_moe_oracle([xf], params, top_k=k, capacity=None, activation=act, routing=[(idx, sc)])
    ref.backward(gy.float())
    rel = lambda a, b: float((a.float() - b).norm() / b.norm().clamp_min(1e-6))   # noqa: E731
    assert rel(y.detach(), ref.detach()) < 1e-2            # bf16 activations and results: 2^-8 each
    assert rel(layer.experts.htoh4.weight.grad, params["htoh4.weight"].grad) < 1.5e-2
    assert rel(layer.experts.h4toh.weight.grad, params["h4toh.weight"].grad) < 1.5e-2
    layer.release()


@pytest.mark.parametrize("act,dtype,k", [("gelu", torch.bfloat16, 2), ("swiglu", torch.float16, 3)])
def test_router_gradients_do_not_depend_on_the_number_of_tokens(act, dtype, k):
    """4095 tokens, and 4096 of which the last has a zero gradient: the logits' gradients are summed in fp32 at any size, so the
    router's gradients are the same bits. (The two-node form rounds them to the element type from 4096 tokens on.)"""
    from ccfuser_b200 import MoEConfig, MoELayer
    torch.manual_seed(k)
    t, d = 4096, 256
    cfg = MoEConfig(d_model=d, d_ffn=512, num_experts=8, top_k=k, activation=act, dtype=dtype, backend="fused", max_tokens=t)
    layer = MoELayer(cfg, device="cuda")
    x = torch.randn(t, d, device="cuda", dtype=dtype)
    gy = torch.randn(t, d, device="cuda", dtype=dtype)
    gy[-1] = 0
    got = []
    for n in (t - 1, t):
        xn = x[:n].clone().requires_grad_()
        for p in layer.parameters():
            p.grad = None
        layer(xn).backward(gy[:n])
        got.append((xn.grad[:t - 1], *(p.grad for p in layer.gate.parameters())))
    layer.check_status()
    for a, b in zip(*got):
        assert torch.equal(a, b)
    layer.release()


_EDGES = [0, 1, 127, 128, 255, 256, 257, 511, 512, 1023, 1024, 1025]


@pytest.mark.parametrize("copies,n", [(1, 256), (1, 1000), (2, 1536), (4, 1536), (8, 1024)])   # 24 to 768 blocks
def test_column_sums_at_the_edges_of_the_sharing_rule(copies, n):
    """Launches of every cluster size (and of none) whose groups keep all, some or one of the blocks; tolerance as above."""
    from ccfuser_b200 import native as N
    rows = _EDGES * copies
    pad = [(r + 127) // 128 * 128 for r in rows]
    base = [sum(pad[:i]) for i in range(len(rows))]
    x = torch.randn(sum(pad), n, device="cuda").bfloat16()
    gb, gr = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (base, rows))
    out = torch.empty(len(rows), n, dtype=torch.bfloat16, device="cuda")
    N.check(N.load().ccf_colsum_grouped(x.data_ptr(), n, n, len(rows), gb.data_ptr(), gr.data_ptr(), out.data_ptr(), 0,
                                        N.stream_ptr()), "ccf_colsum_grouped")
    ref = torch.stack([x[b:b + r].double().sum(0) for b, r in zip(base, rows)])
    mag = torch.stack([x[b:b + r].double().abs().sum(0) for b, r in zip(base, rows)])
    assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * 2.0 ** -16 + 1e-7).all()


@pytest.mark.parametrize("copies,d,k,fp16,hint", [(1, 256, 1, False, 4096), (1, 256, 2, False, 300), (1, 1000, 3, True, 4096),
                                                  (4, 1536, 2, False, 4096), (8, 1024, 2, True, 4096), (1, 256, 1, False, 1)])
def test_router_weight_gradient_at_the_edges_of_the_sharing_rule(copies, d, k, fp16, hint):
    """dWg and db from slot lists of every length (``hint``: the length the launch expects) against fp64: fp32 products and
    sums, one rounding."""
    from ccfuser_b200 import native as N
    dt = torch.float16 if fp16 else torch.bfloat16
    counts = _EDGES * copies
    e, slots = len(counts), (sum(counts) + k - 1) // k * k
    gen = torch.Generator(device="cuda").manual_seed(d)
    order = torch.randperm(slots, device="cuda", generator=gen)[:sum(counts)]
    x = torch.randn(slots // k, d, device="cuda", generator=gen).to(dt)
    g = torch.randn(slots, device="cuda", generator=gen)
    start = [sum(counts[:i]) for i in range(e)]
    raw = torch.zeros(N.MAX_GROUPS + slots, dtype=torch.int32, device="cuda")
    raw[:e] = torch.tensor(start, dtype=torch.int32)
    raw[N.MAX_GROUPS:N.MAX_GROUPS + order.numel()] = order.int()
    cnt = torch.tensor(counts, dtype=torch.int32, device="cuda")
    dw, db = torch.full((e, d), 7.0, dtype=dt, device="cuda"), torch.full((e,), 7.0, dtype=dt, device="cuda")
    N.check(N.load().ccf_router_dw(raw.data_ptr(), cnt.data_ptr(), g.data_ptr(), x.data_ptr(), dw.data_ptr(), db.data_ptr(), hint * e, d,
                                   e, k, int(fp16), N.stream_ptr()), "ccf_router_dw")
    ulp = 2.0 ** (-11 if fp16 else -8)
    for i, (s, c) in enumerate(zip(start, counts)):
        ids = order[s:s + c]
        gs, xs = g[ids].double(), x[ids // k].double()
        ref, mag = gs @ xs, gs.abs() @ xs.abs()
        # the sums of the largest lists stay far below fp16's 65504; 6e-8 is its smallest number
        assert ((dw[i].double() - ref).abs() <= ref.abs() * ulp + mag * 2.0 ** -16 + 1e-7).all(), i
        assert (db[i].double() - gs.sum()).abs() <= gs.sum().abs() * ulp + gs.abs().sum() * 2.0 ** -16 + 1e-7, i


@pytest.mark.parametrize("tiles", [14, 15, 16, 17, 32, 33, 34, 38, 74, 75])
def test_router_where_the_cluster_size_changes(tiles):
    """Token counts on both sides of each step of the rule (clusters of eight, four, two, none)."""
    test_router_splits(128 * tiles - 5, 2048, 64, 2, torch.bfloat16, True)


@pytest.mark.parametrize("world,rank,slots,e,cap", [(2, 0, 100, 8, 20), (2, 1, 1025, 64, 1 << 20), (8, 3, 20000, 64, 300),
                                                   (8, 7, 65536, 256, 1 << 20)])
@pytest.mark.parametrize("device_epoch", [False, True])
def test_route_plan_exchanges_counts_as_the_separate_kernels_do(world, rank, slots, e, cap, device_epoch):
    """One rank's view of a group: the peers' counts and flags are in its table before the launch, so nothing waits; its own
    counts have to appear in every rank's table under the call's epoch. All outputs against ccf_route_ordered + ccf_plan and
    the layout against its definition, with a receive buffer that some rows do not fit."""
    from ccfuser_b200 import native as N
    lib = N.load()
    gen = torch.Generator(device="cuda").manual_seed(slots + rank)
    expert = torch.randint(-1, e + 1, (slots,), dtype=torch.int32, device="cuda", generator=gen)
    others = torch.randint(0, 300, (world, e), dtype=torch.int32, device="cuda", generator=gen)
    i32, epoch, e_loc, nb = dict(dtype=torch.int32, device="cuda"), 5, e // world, (slots + 1023) // 1024
    max_rows = 128 * (2 * e_loc + 1)
    res = []
    for one in (False, True):
        t = {"pos": torch.zeros(slots, **i32), "raw": torch.zeros(e, **i32), "kept": torch.zeros(e, **i32),
             "order_off": torch.zeros(e + 1, **i32), "sorted_slot": torch.full((slots,), -1, **i32),
             "slot_row": torch.zeros(slots, **i32)}
        out = {k: torch.full((n,), -7, **i32) for k, n in (("dst_base", e), ("group_base", e_loc), ("group_rows", e_loc),
                                                          ("local_begin", e_loc), ("local_rows", e_loc), ("sent_rows", 8))}
        out["table_copy"] = torch.full((world, e), -7, **i32)
        tables, flags = torch.full((world, world, e), -7, **i32), torch.zeros(world, 8, **i32)   # what each rank would hold
        tables[rank] = others
        flags[rank, :world] = epoch
        flags[rank, rank] = 0
        status, counter = torch.zeros(2, **i32), torch.full((1,), epoch - 1, **i32)
        p = N.PlanArgs()
        p.count_kept = t["kept"].data_ptr()
        for r in range(world):
            p.peer_table[r], p.peer_flag[r] = tables[r].data_ptr(), flags[r].data_ptr()
        for k, v in out.items():
            setattr(p, k, v.data_ptr())
        p.status, p.wait_limit_ns = status.data_ptr(), 1_000_000_000
        p.world, p.my_rank, p.e_total, p.e_loc, p.epoch, p.max_rows = world, rank, e, e_loc, (0 if device_epoch else epoch), max_rows
        if one:
            N.check(lib.ccf_route_plan(expert.data_ptr(), slots, e, cap, t["pos"].data_ptr(), t["raw"].data_ptr(),
                                       t["kept"].data_ptr(), t["order_off"].data_ptr(), t["sorted_slot"].data_ptr(),
                                       t["slot_row"].data_ptr(), rank * e_loc, None, C.byref(p),
                                       counter.data_ptr() if device_epoch else None, N.stream_ptr()), "ccf_route_plan")
        else:
            bh, bo, ticket = torch.zeros(nb * e, **i32), torch.zeros(nb * e, **i32), torch.zeros(1, **i32)
            N.check(lib.ccf_route_ordered(expert.data_ptr(), slots, e, cap, t["pos"].data_ptr(), bh.data_ptr(), bo.data_ptr(),
                                          t["raw"].data_ptr(), t["kept"].data_ptr(), ticket.data_ptr(),
                                          t["order_off"].data_ptr(), t["sorted_slot"].data_ptr(), t["slot_row"].data_ptr(),
                                          rank * e_loc, N.stream_ptr()), "ccf_route_ordered")
            N.check(lib.ccf_plan_dev_epoch(C.byref(p), counter.data_ptr(), N.stream_ptr()) if device_epoch
                    else lib.ccf_plan(C.byref(p), N.stream_ptr()), "ccf_plan")
        torch.cuda.synchronize()
        assert int(counter) == (epoch if device_epoch else epoch - 1)
        assert (flags[:, rank] == epoch).all() and (tables[:, rank] == t["kept"]).all()
        res.append({**t, **out, "status": status})
    for k in res[0]:
        assert torch.equal(res[0][k], res[1][k]), k
    table = others.cpu().long()
    table[rank] = res[1]["kept"].cpu()
    assert torch.equal(res[1]["table_copy"].cpu().long(), table)
    mine = table[:rank].sum(0)                                       # rows of earlier sources come first
    for o in range(world):
        padded = (table.sum(0)[o * e_loc:(o + 1) * e_loc] + 127) // 128 * 128
        base = torch.cumsum(padded, 0) - padded
        first = base + mine[o * e_loc:(o + 1) * e_loc]
        assert torch.equal(res[1]["dst_base"].cpu().long()[o * e_loc:(o + 1) * e_loc], first)
        assert int(res[1]["sent_rows"][o]) == int(torch.minimum(table[rank, o * e_loc:(o + 1) * e_loc], (max_rows - first).clamp(min=0)).sum())
        if o == rank:
            assert torch.equal(res[1]["group_base"].cpu().long(), base)


@pytest.mark.parametrize("slots", [64, 65536])
def test_route_plan_without_a_peer_ends_with_a_status(slots):
    """A peer whose counts never come: the wait of the cluster's first CTA runs out, the others leave with it, no row is planned."""
    from ccfuser_b200 import native as N
    lib, e, i32 = N.load(), 16, dict(dtype=torch.int32, device="cuda")
    expert = torch.arange(slots, device="cuda", dtype=torch.int32) % e
    pos, row, srt = (torch.zeros(slots, **i32) for _ in range(3))
    raw, kept, off = torch.zeros(e, **i32), torch.zeros(e, **i32), torch.zeros(e + 1, **i32)
    out = {k: torch.full((e,), -7, **i32) for k in ("dst_base", "group_base", "group_rows", "local_begin", "local_rows", "sent_rows")}
    tables, flags, status = torch.zeros(2, 2, e, **i32), torch.zeros(2, 8, **i32), torch.zeros(2, **i32)
    p = N.PlanArgs()
    for r in range(2):
        p.peer_table[r], p.peer_flag[r] = tables[r].data_ptr(), flags[r].data_ptr()
    for k, v in out.items():
        setattr(p, k, v.data_ptr())
    p.status, p.wait_limit_ns = status.data_ptr(), 20_000_000
    p.world, p.my_rank, p.e_total, p.e_loc, p.epoch, p.max_rows = 2, 0, e, e // 2, 1, 1 << 20
    N.check(lib.ccf_route_plan(expert.data_ptr(), slots, e, 1 << 20, pos.data_ptr(), raw.data_ptr(), kept.data_ptr(), off.data_ptr(),
                               srt.data_ptr(), row.data_ptr(), 0, None, C.byref(p), None, N.stream_ptr()), "ccf_route_plan")
    torch.cuda.synchronize()
    assert int(status[0]) & 0xff == 2                   # CCF_ERR_FLAG_TIMEOUT
    assert (out["group_rows"][:e // 2] == 0).all() and (out["sent_rows"][:2] == 0).all() and (out["dst_base"] == 0).all()
    assert (kept == slots // e).all() and torch.equal(pos, torch.arange(slots, device="cuda", dtype=torch.int32) // e)


@pytest.mark.parametrize("a_rows,bn,rows", [(32, 256, [1, 32, 0, 31, 7]), (64, 256, [64, 33, 1, 0])])
@pytest.mark.parametrize("k", [64, 1024])
def test_row_bound_with_mn_major_weights(a_rows, bn, rows, k):
    """The small pipeline geometries with the operand majors of the input-gradient GEMMs (weights read [reduction, columns])."""
    from ccfuser_b200 import native as N
    from ccfuser_b200.ops import gemm as G
    torch.manual_seed(k + len(rows))
    base, acc = [], 0
    for r in rows:
        base.append(acc)
        acc += (r + 127) // 128 * 128
    n, groups = 384, len(rows)
    x = torch.full((max(acc, 128) + 128, k), float("nan"), device="cuda", dtype=torch.bfloat16)
    for b, r in zip(base, rows):
        x[b:b + r] = torch.randn(r, k, device="cuda").bfloat16()
    w = (torch.randn(groups * k, n, device="cuda") * 0.1).bfloat16()
    out = torch.full((x.shape[0], n), 7.0, dtype=torch.bfloat16, device="cuda")
    ws = G.launch(a0=x, b0=w, a_major=N.MAJ_K, b_major=N.MAJ_MN, epi=N.EPI_STORE, n=n, k=k,
                  group_base=torch.tensor(base, dtype=torch.int32, device="cuda"),
                  group_rows=torch.tensor(rows, dtype=torch.int32, device="cuda"), num_groups=groups, b_group_rows=k, out0=out,
                  two_cta=False, bn=bn, a_rows=a_rows)
    ws.check("row bound")
    for i, (b, r) in enumerate(zip(base, rows)):
        ref = x[b:b + r].double() @ w[i * k:(i + 1) * k].double()
        assert ((out[b:b + r].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4).all(), i
        assert (out[b + r:b + (r + 127) // 128 * 128] == 7.0).all()


def _layer_against_oracle(t, d, f, e, k, act, router, tol):
    """Output and every gradient of a layer call against the fp32 oracle on the same routing decisions, with the gate weights
    differentiable through the oracle's router."""
    from ccfuser_b200 import MoEConfig, MoELayer
    from ccfuser_b200.ops.reference import dense_moe_oracle
    torch.manual_seed(t * e + k)
    cfg = MoEConfig(d_model=d, d_ffn=f, num_experts=e, top_k=k, activation=act, dtype=torch.bfloat16, backend="fused",
                    max_tokens=t, router_bias=router != "no bias")
    layer = MoELayer(cfg, device="cuda")
    with torch.no_grad():
        for n, p in layer.named_parameters():
            if n.endswith("bias"):
                p.add_(torch.randn_like(p) * 0.1)
    if router == "frozen weight":
        layer.gate.gate.weight.requires_grad_(False)
    x = torch.randn(t, d, device="cuda", dtype=torch.bfloat16).requires_grad_()
    fm = layer._fused_impl()
    one = fm.one_node(x) is not None
    y = layer(x)
    gy = torch.randn_like(y)
    y.backward(gy)
    layer.check_status()
    with torch.no_grad():
        idx, _ = fm.route(x.detach())
    params = {n.replace("experts.", "").replace("gate.gate.", "gate."): p.detach().float().requires_grad_() for n, p in layer.named_parameters()}
    xf = x.detach().float().requires_grad_()
    logits = torch.nn.functional.linear(xf, params["gate.weight"], params.get("gate.bias"))
    score = torch.softmax(torch.gather(logits, 1, idx.long()), -1)
    (ref,) = dense_moe_oracle([xf], params, top_k=k, capacity=None, activation=act, routing=[(idx, score)])
    ref.backward(gy.float())
    pairs = {"y": (y.detach(), ref.detach()), "x": (x.grad, xf.grad)}
    for n, p in layer.named_parameters():
        if p.requires_grad:
            pairs[n] = (p.grad, params[n.replace("experts.", "").replace("gate.gate.", "gate.")].grad)
        else:
            assert p.grad is None
    layer.release()
    # with one slot per token the gate weight is the constant 1: its router gradients are zero on both sides
    floor = 1e-6 * float(ref.detach().norm())
    bad = {n: err for n, (a, b) in pairs.items() if not (err := float((a.float() - b).norm()) / max(float(b.norm()), floor)) < tol}
    assert not bad, bad
    return one


@pytest.mark.parametrize("t,e,k,act,router", [(1, 16, 2, "gelu", "bias"), (16, 16, 2, "swiglu", "no bias"), (8, 4, 4, "relu", "bias"),
                                             (32, 4, 2, "swiglu", "bias"), (21, 64, 3, "gelu", "frozen weight"),
                                             (60, 8, 1, "swiglu", "bias"), (33, 64, 2, "gelu", "no bias")])
def test_few_token_layer_gradients_match_the_oracle(t, e, k, act, router):
    """Calls whose rows per expert are bounded by 32, by 64 and not at all. Every stored intermediate (pre-activation, activation,
    gate-scaled output, their gradients) is rounded to 8 significant bits, a relative error of at most 2^-8 each and about six on
    the longest path; the router's gradients are differences of two of those."""
    assert _layer_against_oracle(t, 256, 512, e, k, act, router, 6 * 2.0 ** -8)


@pytest.mark.parametrize("t,k", [(32768, 2), (32769, 2)])
def test_layer_around_the_slots_of_the_one_kernel_routing(t, k):
    """65536 slots run as one node, 65538 with the separate routing kernels and two nodes; same tolerance as above."""
    assert _layer_against_oracle(t, 128, 256, 8, k, "gelu", "bias", 6 * 2.0 ** -8) == (t * k <= 65536)


@pytest.mark.parametrize("k", range(0, 10))
@pytest.mark.parametrize("tokens,d", [(1, 8), (300, 72), (513, 2056), (3, 8192)])
def test_combine_reduce_at_every_slot_count(k, tokens, d):
    """Each number of slots per token has its own kernel; blocks end inside tokens, tokens inside blocks. Tolerance as in
    test_combine_reduce."""
    from ccfuser_b200 import native as N
    torch.manual_seed(k + tokens)
    comb = torch.randn(tokens * k + 1, d, device="cuda").bfloat16()[:tokens * k]
    row = torch.randint(-1, 5, (tokens * k + 1,), dtype=torch.int32, device="cuda")[:tokens * k]
    comb[row < 0] = float("nan")
    guard = torch.full((tokens + 1, d), 7.0, dtype=torch.bfloat16, device="cuda")
    N.check(N.load().ccf_combine_reduce(comb.data_ptr(), row.data_ptr(), guard.data_ptr(), tokens, k, d, 0, N.stream_ptr()),
            "ccf_combine_reduce")
    ref = torch.where((row >= 0).unsqueeze(1), comb.double(), torch.zeros((), dtype=torch.float64, device="cuda")).view(tokens, k, d).sum(1)
    assert ((guard[:tokens].double() - ref).abs() <= ref.abs() * 2.0 ** -8 * 1.01 + 1e-6).all()
    assert (guard[tokens] == 7.0).all()
