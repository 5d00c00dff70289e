"""pg_moe_products (grouped tcgen05 products over the routing plan) against 64-bit products of the same rows.

Bounds: the activations between the products are bf16 (2^-8 of the value that is rounded; the silu / relu^2 slope carries the sum's error), sums are fp32."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu

ACTS = {seq_ops.ACT_NONE: lambda z: z, seq_ops.ACT_RELU2: lambda z: z.clamp(min=0) ** 2, seq_ops.ACT_GELU_ERF: torch.nn.functional.gelu}


@pytest.mark.parametrize("T,top,n", [(1, 1, 1), (1, 4, 9), (5, 2, 3), (16, 4, 6), (17, 3, 40), (64, 2, 2), (65, 1, 3), (300, 4, 14), (700, 2, 5)])
@pytest.mark.parametrize("D,F", [(64, 8), (136, 200), (2048, 1024), (72, 520)])
@pytest.mark.parametrize("act", [seq_ops.ACT_NONE, seq_ops.ACT_RELU2, seq_ops.ACT_GELU_ERF, seq_ops.ACT_SILU_GLU])
def test_against_64_bits(T, top, n, D, F, act):
    g = torch.Generator(device="cuda").manual_seed(T * 31 + D + act)
    ids = torch.stack([torch.randperm(n + 1, generator=g, device="cuda")[:top] for _ in range(T)]).to(torch.int32)  # id n: an identity output, no row
    counts = torch.bincount(ids[ids < n].long(), minlength=n).to(torch.int32)
    plan = seq_ops.MoePlan(ids.contiguous(), counts, n)
    glu = act == seq_ops.ACT_SILU_GLU
    x = torch.randn(T, D, generator=g, device="cuda").bfloat16()
    up = (torch.randn(n, 2 * F if glu else F, D, generator=g, device="cuda") * D ** -0.5).bfloat16()
    down = (torch.randn(n, D, F, generator=g, device="cuda") * F ** -0.5).bfloat16()
    xg, mid = torch.empty(plan.pairs, D, device="cuda", dtype=torch.bfloat16), torch.empty(plan.pairs, F, device="cuda", dtype=torch.bfloat16)
    eo = torch.full((plan.pairs, D), float("nan"), device="cuda")
    seq_ops.moe_products(x, plan, up, down, xg, mid, eo, act)
    for t in range(T):
        for k in range(top):
            e, row = int(ids[t, k]), int(plan.pair_row[t * top + k])
            if e >= n:
                assert row == -1
                continue
            if t % 7 and T > 64:
                continue
            z = up[e].double() @ x[t].double()
            if glu:
                want = z[0::2] * torch.sigmoid(z[0::2]) * z[1::2]
                slope = z.abs().view(-1, 2).amax(1) + 1
            else:
                want, slope = ACTS[act](z), 2 * z.abs() + 2
            err = 2.0 ** -8 * want.abs() + 2.0 ** -18 * slope ** 2
            assert ((mid[row].double() - want).abs() <= err).all()
            got = down[e].double() @ mid[row].double()
            assert ((eo[row].double() - got).abs() <= 2.0 ** -20 * (down[e].double().abs() @ mid[row].double().abs()) + 1e-30).all()


@pytest.mark.parametrize("T,top,n", [(16, 4, 2), (32, 3, 2), (48, 4, 2)])
def test_one_token_may_choose_an_expert_again(T, top, n):
    """A token whose router scores are NaN takes expert 0 every time: that expert then owns more rows than the step has tokens, and the other tokens' rows are
    what they are without it."""
    D, F = 64, 72
    logits = torch.randn(T, max(n, top), device="cuda")
    logits[0] = float("nan")
    ids, _, counts = seq_ops.moe_route(logits, None, n, top, 1, 1, 1.0)
    plan = seq_ops.MoePlan(ids, counts, n)
    assert int(counts.max()) > T
    x = torch.randn(T, D, device="cuda").bfloat16()
    up, down = torch.randn(n, F, D, device="cuda").bfloat16(), torch.randn(n, D, F, device="cuda").bfloat16()
    xg, mid = torch.empty(plan.pairs, D, device="cuda", dtype=torch.bfloat16), torch.empty(plan.pairs, F, device="cuda", dtype=torch.bfloat16)
    eo = torch.full((plan.pairs, D), float("nan"), device="cuda")
    seq_ops.moe_products(x, plan, up, down, xg, mid, eo, seq_ops.ACT_NONE)
    for t in range(T):
        for k in range(top):
            e, row = int(ids[t, k]), int(plan.pair_row[t * top + k])
            if e >= n:
                continue
            z = up[e].double() @ x[t].double()
            assert ((mid[row].double() - z).abs() <= 2.0 ** -8 * z.abs() + 2.0 ** -18 * (up[e].double().abs() @ x[t].double().abs())).all()
            got = down[e].double() @ mid[row].double()
            assert ((eo[row].double() - got).abs() <= 2.0 ** -20 * (down[e].double().abs() @ mid[row].double().abs()) + 1e-30).all()


@pytest.mark.parametrize("T,top,n", [(3, 2, 2), (70, 3, 4)])
def test_rows_next_to_a_tile_stay_out(T, top, n):
    """Scratch rows that no expert owns hold anything, an infinity in one token's row and a NaN in one expert's weights stay with their rows."""
    D, F = 72, 136
    ids = torch.stack([torch.randperm(n + 1, device="cuda")[:top] for _ in range(T)]).to(torch.int32).contiguous()  # id n: no row
    ids[0, 0], ids[0, 1:] = n, torch.arange(top - 1, device="cuda")
    counts = torch.bincount(ids[ids < n].long(), minlength=n).to(torch.int32)
    plan = seq_ops.MoePlan(ids, counts, n)
    x = torch.randn(T, D, device="cuda").bfloat16()
    up, down = (torch.randn(n, F, D, device="cuda") * D ** -0.5).bfloat16(), (torch.randn(n, D, F, device="cuda") * F ** -0.5).bfloat16()
    x[1, 5], down[n - 1, D - 1, 3] = float("inf"), float("nan")
    b = dict(device="cuda", dtype=torch.bfloat16)
    xg, mid = torch.full((plan.pairs, D), float("nan"), **b), torch.full((plan.pairs, F), float("nan"), **b)
    eo = torch.zeros(plan.pairs, D, device="cuda")
    seq_ops.moe_products(x, plan, up, down, xg, mid, eo, seq_ops.ACT_RELU2)
    owned = 0
    for t in range(T):
        for k in range(top):
            e, row = int(ids[t, k]), int(plan.pair_row[t * top + k])
            if e >= n:
                continue
            owned += 1
            last = D - 1 if e == n - 1 else D
            if t != 1:
                assert eo[row, :last].isfinite().all() and mid[row].isfinite().all()
                got = down[e, :last].double() @ mid[row].double()
                assert ((eo[row, :last].double() - got).abs() <= 2.0 ** -20 * (down[e, :last].double().abs() @ mid[row].double().abs()) + 1e-30).all()
            if e == n - 1:
                assert eo[row, D - 1].isnan()
    assert owned < plan.pairs and not eo[owned:].any()


@pytest.mark.parametrize("D,F,T", [(128, 64, 5), (128, 128, 5), (128, 128, 300), (256, 256, 5), (256, 256, 300)])
@pytest.mark.parametrize("activation", ["relu2", "silu_glu"])
def test_both_sides_of_the_line(D, F, T, activation):
    """Whichever kernels a routed feed-forward takes for its size, its rows are those of the products that gather on the way."""
    from paligemma_multimodal_system_b200 import mixers
    prec, n, top = seq_ops.Precision(torch.bfloat16), 4, 2
    ff = mixers.RoutedFeedForward(D, n, 0, top, 1, 1, 1.0, F, 0, activation=activation, correction=False)
    ff.load(lambda name, shape: torch.randn(*shape, device="cuda") * shape[-1] ** -0.5, "")
    ff.pack(prec)
    ids = torch.stack([torch.randperm(n, device="cuda")[:top] for _ in range(T)]).to(torch.int32).contiguous()
    counts = torch.bincount(ids.flatten().long(), minlength=n).to(torch.int32)
    plan = seq_ops.MoePlan(ids, counts, n)
    h = torch.randn(T, D, device="cuda").bfloat16()
    eo = ff.expert_products(h, plan, counts, prec)
    mid = seq_ops.moe_gemm(h, plan, ff.w_up, prec.empty(plan.pairs, F), gather=True, act=ff.act)
    want = seq_ops.moe_gemm(mid, plan, ff.w_down, torch.empty(plan.pairs, D, device="cuda"), gather=False)
    # activations that round to neighbouring bf16 values: 2^-8 of each, F of them with weights of about F^-0.5
    assert (eo - want).abs().max() <= 2.0 ** -7 * mid.float().abs().max()


@pytest.mark.parametrize("D,F,T", [(128, 64, 520), (1024, 512, 900), (2048, 2048, 700)])  # the last: above 1.2e9 multiply-adds a run
@pytest.mark.parametrize("activation", ["relu2", "silu_glu"])
def test_dense_runs(D, F, T, activation):
    """Long runs as dense products side by side, the small ones on the persistent kernels and the large ones clustered: the rows of the products that gather on the way."""
    from paligemma_multimodal_system_b200 import mixers
    prec, n = seq_ops.Precision(torch.bfloat16), 2
    ff = mixers.RoutedFeedForward(D, n, 0, 1, 1, 1, 1.0, F, 0, activation=activation, correction=False)
    ff.load(lambda name, shape: torch.randn(*shape, device="cuda") * shape[-1] ** -0.5, "")
    ff.pack(prec)
    ids = (torch.rand(T, 1, device="cuda") < 0.4).to(torch.int32)
    counts = torch.bincount(ids.flatten().long(), minlength=n).to(torch.int32)
    plan = seq_ops.MoePlan(ids, counts, n)
    h = torch.randn(T, D, device="cuda").bfloat16()
    assert ff._dense_segments(T, prec)
    eo = ff.expert_products(h, plan, counts, prec)
    mid = seq_ops.moe_gemm(h, plan, ff.w_up, prec.empty(plan.pairs, F), gather=True, act=ff.act)
    want = seq_ops.moe_gemm(mid, plan, ff.w_down, torch.empty(plan.pairs, D, device="cuda"), gather=False)
    assert (eo - want).abs().max() <= 2.0 ** -7 * mid.float().abs().max()


@pytest.mark.parametrize("T,top,n_all,n_real,nan", [(1, 1, 1, 1, False), (1, 4, 14, 14, False), (300, 4, 16, 14, False), (1024, 4, 14, 14, False), (819, 5, 1100, 1024, False),
                                                    (256, 4, 40, 33, True), (64, 8, 64, 1, False)])
def test_plan_of_few_pairs(T, top, n_all, n_real, nan):
    """Counters, plan and scatter in one launch against the three: the same choices, runs and tiles, and every pair on a row of its expert's run."""
    logits = torch.randn(T, n_all, device="cuda")
    if nan:
        logits[::3] = float("nan")  # (a token that chooses expert 0 every time)
    ids, wts, counts = seq_ops.moe_route(logits, None, n_real, top, 1, 1, 1.0)
    ref = seq_ops.MoePlan(ids, counts, n_real)
    ids2, wts2 = torch.empty_like(ids), torch.empty_like(wts)
    offsets, plan, order, row = (torch.full_like(t, -7) for t in (ref.offsets, ref.plan, ref.sorted_pair, ref.pair_row))
    _lib.check(_lib.lib().pg_moe_route_plan(logits.data_ptr(), n_all, 0, ids2.data_ptr(), wts2.data_ptr(), offsets.data_ptr(), plan.data_ptr(), order.data_ptr(), row.data_ptr(), T, n_all,
                                            n_real, top, 1, 1, 1.0, 0, 0, ref.max_tiles, _lib.stream()), "plan")
    assert torch.equal(ids, ids2) and torch.equal(wts.view(torch.int32), wts2.view(torch.int32)) and torch.equal(offsets, ref.offsets)
    tiles = int(ref.plan[0])
    assert torch.equal(plan[4:4 + 3 * tiles], ref.plan[4:4 + 3 * tiles]) and int(plan[0]) == tiles
    flat, total = ids.flatten(), int(offsets[n_real])
    real = flat < n_real
    assert (row[~real] == -1).all() and torch.equal(row[real].sort().values, torch.arange(total, device="cuda", dtype=torch.int32))
    assert torch.equal(order[row[real].long()], torch.nonzero(real).flatten().int())
    e = flat[real].long()
    assert (row[real] >= offsets[e]).all() and (row[real] < offsets[e + 1]).all()


def test_plan_of_too_many_pairs_is_refused():
    z, i = torch.zeros(1025, 4, device="cuda"), torch.zeros(4100, device="cuda", dtype=torch.int32)
    for T, n in ((1025, 4), (4, 0), (4, 1025)):
        assert _lib.lib().pg_moe_route_plan(z.data_ptr(), 4, 0, i.data_ptr(), z.data_ptr(), i.data_ptr(), i.data_ptr(), i.data_ptr(), i.data_ptr(), T, max(4, n), n, 4, 1, 1, 1.0, 0, 0, 99,
                                            _lib.stream()) != 0
