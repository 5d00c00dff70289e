"""Prompt attention on tensor memory where it can go wrong -- tiles of 128 rows and 64 keys, windows and kept first keys, every optional part of the score, pages whose
unused rows hold NaNs -- against 64-bit sums.  Scores are sums of bf16 products in fp32 and probabilities keep 24 bits, so a result differs by its rounding to bf16
(2^-9, bound 2^-8) and about 1e-5 of the values' scale; tanh32 adds 2e-7 of the cap to a score."""
import math

import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


def _t(*shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


def _want(q, k, v, first, scale, softcap, window, keep, hs, sink):
    """q [n, H, dim] at positions first .., k / v [L, G, .], in 64 bits."""
    n, H, _ = q.shape
    G, L = k.shape[1], k.shape[0]
    kk, vv = (t.double().repeat_interleave(H // G, 1) for t in (k, v))
    s = torch.einsum("ihd,jhd->hij", q.double(), kk) * scale
    if hs is not None:
        s = s * hs.double()[:, None, None]
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    i, j = torch.arange(first, first + n, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    s = s.masked_fill(~((j <= i) & ((i - j < window) | (j < keep)) if window else j <= i), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(H, n, 1)], -1)
    return torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :L], vv)


@pytest.mark.parametrize("dim,vdim,G,gsz", [(64, 64, 2, 4), (96, 64, 3, 1), (128, 128, 1, 4), (64, 128, 2, 3), (128, 64, 1, 5), (64, 64, 1, 129)])
@pytest.mark.parametrize("ns,ctxs", [((2, 1, 33, 130), (0, 5, 63, 200)), ((300,), (0,)), ((64, 65), (64, 127)), ((5,), (1000,))])
@pytest.mark.parametrize("window,keep", [(0, 0), (33, 0), (70, 5), (1, 1), (512, 130)])
def test_masks(dim, vdim, G, gsz, ns, ctxs, window, keep):
    _run(dim, vdim, G, gsz, ns, ctxs, window, keep)


@pytest.mark.parametrize("dim,vdim", [(64, 64), (96, 64), (128, 128)])
@pytest.mark.parametrize("opts", [dict(softcap=5.0), dict(hs=True), dict(sink=True), dict(gate="row"), dict(gate="head"), dict(ld=True), dict(softcap=3.0, hs=True, sink=True, gate="head", ld=True),
                                  dict(scale=-0.1), dict(big=True)])
def test_options(dim, vdim, opts):
    _run(dim, vdim, 2, 2, (70, 1, 129), (0, 9, 77), 100, 3, **opts)


@pytest.mark.parametrize("ns,ctxs", [((2, 1, 33, 130), (0, 5, 63, 200)), ((300,), (0,)), ((64, 65), (64, 127)), ((5,), (1000,))])
@pytest.mark.parametrize("window,keep", [(0, 0), (33, 0), (70, 5), (512, 130)])
def test_masks_of_many_heads(ns, ctxs, window, keep):
    """Heads of 64 / 128 in more CTAs than SMs (fewer stay with mma.sync, as do a handful of rows in many CTAs)."""
    _run(64, 128, 160, 1, ns, ctxs, window, keep)


@pytest.mark.parametrize("n", [1, 4, 5])
def test_either_side_of_a_handful_of_rows(n):
    _run(64, 64, 40, 4, (n, 2, n, 1), (70, 0, 300, 5), 0, 0)  # 16 and 20 rows in 160 CTAs


@pytest.mark.parametrize("dim,vdim,G,gsz", [(64, 64, 2, 4), (96, 64, 3, 1), (128, 64, 1, 5)])
@pytest.mark.parametrize("ns,ctxs", [((130, 1, 3), (1000, 5, 0)), ((300,), (500,)), ((2, 65), (511, 800)), ((790,), (0,))])
@pytest.mark.parametrize("window,keep", [(0, 0), (700, 5), (600, 130), (64, 1000)])
@pytest.mark.parametrize("opts", [dict(), dict(softcap=3.0, hs=True, sink=True, gate="row", big=True)])
def test_keys_shared_out_over_two_ctas(dim, vdim, G, gsz, ns, ctxs, window, keep, opts):
    """Few blocks with many tiles: odd and even halves, blocks of a single tile whose second CTA has none, halves on both sides of the gap in front of a window."""
    _run(dim, vdim, G, gsz, ns, ctxs, window, keep, **opts)


@pytest.mark.parametrize("dim,vdim,G,gsz", [(64, 64, 2, 4), (96, 64, 3, 1), (128, 128, 1, 2)])
@pytest.mark.parametrize("at", [0, 31, 32, 69])
def test_portions_among_many_single_tokens(dim, vdim, G, gsz, at):
    """Single tokens left to another kernel: the entries with rows are found by their number among 32, 64 and more."""
    ns, ctxs = [1] * 70, [0] * 70
    ns[at], ctxs[at], ns[(at + 33) % 70], ctxs[(at + 33) % 70] = 200, 40, 3, 90
    _run(dim, vdim, G, gsz, ns, ctxs, 0, 0, skip=True)


def _run(dim, vdim, G, gsz, ns, ctxs, window, keep, softcap=0.0, hs=False, sink=False, gate=None, ld=False, scale=None, big=False, skip=False):
    H, scale = G * gsz, dim ** -0.5 if scale is None else scale
    rows, first = [], 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        p = (n + c + 63) // 64
        rows.append(dict(tokens=[1] * n, ctx=c, slot=i, pages=list(range(first, first + p))[::-1]))
        first += p
    b = seq_ops.make_step_batch(rows)
    kp = torch.full((first, 64, G * dim), float("nan"), device="cuda", dtype=torch.bfloat16)
    vp = torch.full((first, 64, G * vdim), float("nan"), device="cuda", dtype=torch.bfloat16)
    q = _t(b.T, H * dim, seed=1) * (30 if big else 1)  # (big: maxima that grow from tile to tile)
    ks, vs = [], []
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        k, v = _t(n + c, G * dim, seed=10 + i), _t(n + c, G * vdim, seed=20 + i)
        if big:
            k = (k * torch.linspace(0.1, 3, n + c, device="cuda")[:, None]).to(torch.bfloat16)
        for j, p in enumerate(rows[i]["pages"]):
            part = slice(64 * j, min(64 * j + 64, n + c))
            kp[p, : part.stop - part.start], vp[p, : part.stop - part.start] = k[part], v[part]
        ks.append(k.view(-1, G, dim))
        vs.append(v.view(-1, G, vdim))
    hst = torch.linspace(-0.7, 1.5, H, device="cuda") if hs else None
    skt = torch.linspace(-2, 3, H, device="cuda") if sink else None
    pitch = H * vdim + 8 if ld else H * vdim
    out = torch.full((b.T, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
    g = None if gate is None else _t(b.T, H if gate == "head" else H * vdim, seed=5)
    score = seq_ops.ScoreOptions(H, window or None, keep, sink=skt, head_scale=hst, out_scale=0.5 if ld else 1.0, out_ld=pitch if ld else 0)
    seq_ops.attn_ragged(q, kp, vp, g, out, b, H, G, dim, vdim, scale, softcap, 64, gate_per_head=gate == "head", score=score, decode_kernel=False, skip_singles=skip)
    r = 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        want = _want(q[r:r + n].view(n, H, dim), ks[i], vs[i], c, scale, softcap, window, keep, hst, skt) * (0.5 if ld else 1.0)
        if g is not None:
            want = want * torch.sigmoid(g[r:r + n].double()).view(n, H, -1)
        got = out[r:r + n, : H * vdim].double().view(n, H, vdim)
        if skip and n == 1:
            assert (got == 7).all()
        else:
            assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + (2e-4 if big else 5e-5)).all(), (i, (got - want).abs().max().item())
        r += n
    if ld:
        assert (out[:, H * vdim:] == 7).all()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dim,vdim,G,gsz,window,keep", [(64, 64, 2, 4, 0, 0), (64, 64, 1, 1, 0, 0), (128, 128, 1, 4, 0, 0), (96, 64, 2, 1, 70, 0), (64, 128, 16, 2, 33, 40),
                                                        (128, 64, 1, 129, 0, 0), (64, 64, 3, 2, 90, 5)])
@pytest.mark.parametrize("opts", [dict(), dict(softcap=5.0, hs=True, sink=True, gate="head", ld=True), dict(gate="row")])
@pytest.mark.parametrize("n", [300, 800])
def test_values_that_are_not_finite(dim, vdim, G, gsz, window, keep, opts, bad, n):
    """A broken value reaches the rows that see it and no others: not those before it in their block, nor those whose window begins behind it."""
    ctx, at = 30, 207
    H, L, softcap = G * gsz, ctx + n, opts.get("softcap", 0.0)
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=ctx, slot=0, pages=list(range((L + 63) // 64)))])
    kp, vp = (_t((L + 63) // 64, 64, G * d, seed=s) for d, s in ((dim, 2), (vdim, 3)))
    vp[at // 64, at % 64] = bad
    pitch = H * vdim + (8 if "ld" in opts else 0)
    q, out = _t(n, H * dim, seed=1), torch.full((n, pitch), 7.0, device="cuda", dtype=torch.bfloat16)
    hs = torch.linspace(-0.7, 1.5, H, device="cuda") if "hs" in opts else None
    sink = torch.linspace(-2, 3, H, device="cuda") if "sink" in opts else None
    gate = opts.get("gate")
    g = None if gate is None else _t(n, H if gate == "head" else H * vdim, seed=5)
    score = seq_ops.ScoreOptions(H, window or None, keep, sink=sink, head_scale=hs, out_scale=0.5 if "ld" in opts else 1.0, out_ld=pitch if "ld" in opts else 0)
    seq_ops.attn_ragged(q, kp, vp, g, out, b, H, G, dim, vdim, dim ** -0.5, softcap, 64, gate_per_head=gate == "head", score=score, decode_kernel=False)
    k, v = kp.view(-1, G, dim)[:L], vp.view(-1, G, vdim)[:L].clone()
    v[at] = 0
    want = _want(q.view(n, H, dim), k, v, ctx, dim ** -0.5, softcap, window, keep, hs, sink) * (0.5 if "ld" in opts else 1.0)
    if g is not None:
        want = want * torch.sigmoid(g.double()).view(n, H, -1)
    pos = torch.arange(ctx, L, device="cuda")
    sees = (pos >= at) & (pos - at < window) if window else pos >= at  # (207 is none of the kept first keys)
    got = out[:, : H * vdim].double().view(n, H, vdim)
    assert (~torch.isfinite(got[sees])).all()
    assert ((got[~sees] - want[~sees]).abs() <= want[~sees].abs() * 2.0 ** -8 + 5e-5).all()
    if pitch > H * vdim:
        assert (out[:, H * vdim:] == 7).all()


@pytest.mark.parametrize("page", [8, 16, 32, 128, 192])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128)])
def test_page_sizes(page, dim, vdim):
    """A tile of 64 keys as several pages, the last of them missing, and as part of a page."""
    G, gsz, ns, ctxs, window, keep = 2, 2, (70, 1, 9, 130), (0, 5, 63, 200), 100, 3
    H, rows, first = G * gsz, [], 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        p = (n + c + page - 1) // page
        rows.append(dict(tokens=[1] * n, ctx=c, slot=i, pages=list(range(first, first + p))[::-1] + [0] * ((n + c + 63) // 64 - p)))  # (at least one a 64 keys is asked for)
        first += p
    b = seq_ops.make_step_batch(rows)
    kp, vp = (torch.full((first, page, G * d), float("nan"), device="cuda", dtype=torch.bfloat16) for d in (dim, vdim))
    q, out, ks, vs = _t(b.T, H * dim, seed=1), torch.full((b.T, H * vdim), 7.0, device="cuda", dtype=torch.bfloat16), [], []
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        k, v = _t(n + c, G * dim, seed=10 + i), _t(n + c, G * vdim, seed=20 + i)
        for j, p in enumerate(rows[i]["pages"][: (n + c + page - 1) // page]):
            part = slice(page * j, min(page * j + page, n + c))
            kp[p, : part.stop - part.start], vp[p, : part.stop - part.start] = k[part], v[part]
        ks.append(k.view(-1, G, dim))
        vs.append(v.view(-1, G, vdim))
    seq_ops.attn_ragged(q, kp, vp, None, out, b, H, G, dim, vdim, dim ** -0.5, 0.0, page, score=seq_ops.ScoreOptions(H, window, keep), decode_kernel=False)
    r = 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        want = _want(q[r:r + n].view(n, H, dim), ks[i], vs[i], c, dim ** -0.5, 0.0, window, keep, None, None)
        got = out[r:r + n].double().view(n, H, vdim)
        assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 5e-5).all(), (i, (got - want).abs().max().item())
        r += n


@pytest.mark.parametrize("dim,vdim,G,gsz", [(64, 64, 2, 4), (96, 64, 3, 1), (128, 128, 1, 2), (192, 128, 1, 3), (32, 32, 2, 2)])
@pytest.mark.parametrize("skip", [0, 1])
def test_what_the_host_has_counted_changes_nothing(dim, vdim, G, gsz, skip):
    """pg_attn_ragged_mma knows nothing of the batch; with the number of entries that have rows, the same bits (short contexts: the keys of a block stay with one CTA)."""
    from paligemma_multimodal_system_b200 import _lib
    ns, ctxs, H = [1, 200, 1, 1, 70, 1], [90, 40, 5, 300, 0, 64], G * gsz
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=c, slot=i, pages=[(7 * i + j) % 11 for j in range((n + c + 63) // 64)]) for i, (n, c) in enumerate(zip(ns, ctxs))])
    q, kp, vp = _t(b.T, H * dim, seed=1), _t(11, 64, G * dim, seed=2), _t(11, 64, G * vdim, seed=3)
    L, outs = _lib.lib(), []
    for counted in (None, 0, 2 if skip else len(ns), len(ns)):
        out = torch.full((b.T, H * vdim), 7.0, device="cuda", dtype=torch.bfloat16)
        args = [q.data_ptr(), kp.data_ptr(), vp.data_ptr(), 0, 0, out.data_ptr(), b.row0.data_ptr(), b.n.data_ptr(), b.ctx.data_ptr(), b.page_table.data_ptr(), b.max_pages, 64, len(ns),
                b.max_n, H, G, dim, vdim, dim ** -0.5, 0.0, skip, 0]
        if counted is None:
            _lib.check(L.pg_attn_ragged_mma(*args, 0, _lib.stream()), "pg_attn_ragged_mma")
        else:
            _lib.check(L.pg_attn_ragged_mma_sized(*args, counted, 240, 0, _lib.stream()), "pg_attn_ragged_mma_sized")
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs) and (outs[0] == 7).all(1).sum() == (4 if skip else 0)


@pytest.mark.parametrize("dim,vdim,G,gsz,n,ctx", [(64, 64, 8, 4, 4, 300), (64, 64, 16, 1, 2, 900), (64, 128, 16, 1, 200, 40), (64, 128, 16, 1, 200, 100), (64, 128, 4, 4, 70, 600)])
@pytest.mark.parametrize("many", [0, 40])
def test_a_few_rows_beside_single_tokens(dim, vdim, G, gsz, n, ctx, many):
    """Single tokens left to another kernel are no CTAs of this one: the form is that of the portion alone, on either side of the lines between the two kernels."""
    _run(dim, vdim, G, gsz, [1] * (many // 2) + [n] + [1] * (many // 2), [70] * (many // 2) + [ctx] + [0] * (many // 2), 0, 0, skip=True)
