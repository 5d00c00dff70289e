"""The short convolution that takes several rows of 4 or 8 adjacent channels a lane: runs of rows and their remainders, one to three sections, groups of one lane to a warp, normed
and plain, continued and fresh slots, against 64 bits."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu

SECTIONS = [
    [dict(groups=4, size=64, unit=True, scale=0.5), dict(groups=4, size=64, unit=True), dict(groups=4, size=64)],
    [dict(groups=3, size=8, unit=True), dict(groups=2, size=16, unit=True), dict(groups=1, size=128, unit=True)],
    [dict(groups=5, size=4, total=20)],
    [dict(groups=2, size=256, unit=True), dict(groups=9, size=32, total=264)],
]


@pytest.mark.parametrize("sections", SECTIONS)
@pytest.mark.parametrize("taps", [1, 2, 4, 7])
@pytest.mark.parametrize("ns,ctxs", [((1, 2, 3, 4, 5), (0, 9, 0, 2, 7)), ((17, 64, 130), (0, 5, 1)), ((700,) * 40, (0,) * 40)])
@pytest.mark.parametrize("bias", [False, True])
def test_rows(sections, taps, ns, ctxs, bias):
    secs, C, X = [], 0, 8
    for s in sections:
        total = s.get("total", s["groups"] * s["size"])
        secs.append(dict(s, xcol=X, ccol=C))
        C, X = C + (total + 7) // 8 * 8, X + (total + 7) // 8 * 8 + 16
    cs = seq_ops.ConvSections(secs)
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=c, slot=i, pages=list(range((n + c + 63) // 64))) for i, (n, c) in enumerate(zip(ns, ctxs))])
    g = torch.Generator(device="cuda").manual_seed(taps)
    x = torch.randn(b.T, X, generator=g, device="cuda").to(torch.bfloat16)
    w, bs = torch.randn(taps, C, generator=g, device="cuda") * 0.5, torch.randn(C, generator=g, device="cuda") if bias else None
    state = torch.randn(len(ns), taps - 1, C, generator=g, device="cuda").to(torch.bfloat16).float() if taps > 1 else None
    before = None if state is None else state.clone()
    out = torch.full((b.T, C), 7.0, device="cuda", dtype=torch.bfloat16)
    inv = torch.zeros(b.T, cs.unit_groups, device="cuda") if cs.unit_groups else None
    seq_ops.short_conv(x, w, state, out, cs, b, bias=bs, inv=inv)
    r = 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        if i >= 3 and n == 700:  # (three of the equal ones)
            break
        u = 0
        for s in secs:
            total = s.get("total", s["groups"] * s["size"])
            xs, cols = x[r:r + n, s["xcol"]:s["xcol"] + total].double(), slice(s["ccol"], s["ccol"] + total)
            old = torch.zeros(taps - 1, total, device="cuda", dtype=torch.float64) if taps > 1 and c == 0 else (before[i, :, cols].double() if taps > 1 else xs[:0])
            full = torch.cat([old, xs])
            y = sum(w[j, cols].double() * full[j:j + n] for j in range(taps)) + (bs[cols].double() if bias else 0)
            y = y * torch.sigmoid(y)
            got = out[r:r + n, cols].double()
            # silu by the hardware exponential: 2^-18 of a value of a sum of up to 7 products below 4 each; then one rounding to bf16
            assert ((got - y).abs() <= 2.0 ** -8 * y.abs() + 2.0 ** -14).all()
            if taps > 1:
                assert torch.equal(state[i, :, cols].double(), full[n:])
            if s.get("unit"):
                # the norm is that of the stored activations: fp32 sums of up to 256 squares
                want = s.get("scale", 1.0) / torch.sqrt((got.view(n, s["groups"], s["size"]) ** 2).sum(-1) + 1e-6)
                assert ((inv[r:r + n, u:u + s["groups"]].double() - want).abs() <= 2.0 ** -18 * want).all()
                u += s["groups"]
        r += n


@pytest.mark.parametrize("n,many", [(100, 40), (700, 40), (700, 3), (64, 300)])
def test_how_rows_are_shared_out_changes_nothing(n, many):
    """pg_short_conv knows nothing of the batch; told how many entries are more than single tokens it takes other runs of rows, and the same bits come out."""
    import ctypes as C
    from paligemma_multimodal_system_b200 import _lib
    ns = [1] * (many // 2) + [n] + [1] * (many - many // 2)
    b = seq_ops.make_step_batch([dict(tokens=[1] * k, ctx=i % 5, slot=i, pages=list(range(12))) for i, k in enumerate(ns)])
    cs = seq_ops.ConvSections([dict(groups=8, size=64, xcol=0, ccol=0, unit=True), dict(groups=4, size=64, xcol=512, ccol=512)])
    g = torch.Generator(device="cuda").manual_seed(n)
    x, w, state = torch.randn(b.T, 768, generator=g, device="cuda").to(torch.bfloat16), torch.randn(4, 768, generator=g, device="cuda"), torch.randn(len(ns), 3, 768, generator=g, device="cuda")
    res, L = [], _lib.lib()
    for portions in (None, 0, 1, len(ns)):
        st, out, inv = state.clone(), torch.full_like(x, 7.0), torch.zeros(b.T, 8, device="cuda")
        args = [x.data_ptr(), 768, w.data_ptr(), 0, st.data_ptr(), out.data_ptr(), 768, inv.data_ptr(), 8, C.addressof(cs.c), 4, 768, b.row0.data_ptr(), b.n.data_ptr(), b.ctx.data_ptr(),
                b.slot.data_ptr(), len(ns), n]
        if portions is None:
            _lib.check(L.pg_short_conv(*args, 0, _lib.stream()), "pg_short_conv")
        else:
            _lib.check(L.pg_short_conv_sized(*args, portions, 0, _lib.stream()), "pg_short_conv_sized")
        res.append((out, st, inv))
    for r in res[1:]:
        assert all(torch.equal(a, c) for a, c in zip(r, res[0]))
