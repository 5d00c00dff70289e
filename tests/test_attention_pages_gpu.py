"""pg_attn_ragged_mma reads a tile of 64 keys through one page lookup when pages hold 64 rows and row by row otherwise: the same rows under another
page size give the same bits."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page", [16, 32, 128, 192])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (96, 64), (192, 128), (32, 32)])
@pytest.mark.parametrize("n,ctx", [(1, 0), (5, 60), (64, 0), (70, 131), (200, 184)])
def test_other_page_sizes(page, dim, vdim, n, ctx):
    H, G, rows = 4, 2, 384
    q = torch.randn(n, H * dim, device="cuda").bfloat16()
    k, v = torch.randn(rows, G * dim, device="cuda").bfloat16(), torch.randn(rows, G * vdim, device="cuda").bfloat16()
    outs = []
    for size in (64, page):
        b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=ctx, slot=0, pages=list(range(6)))])
        order = torch.randperm(rows // size, device="cuda")
        kp, vp = torch.empty(rows // size, size, G * dim, device="cuda", dtype=torch.bfloat16), torch.empty(rows // size, size, G * vdim, device="cuda", dtype=torch.bfloat16)
        kp[order], vp[order] = k.view(-1, size, G * dim), v.view(-1, size, G * vdim)
        b.page_table, b.max_pages, b.singles = order.to(torch.int32).view(1, -1).contiguous(), rows // size, 0
        out = torch.full((n, H * vdim), float("nan"), device="cuda", dtype=torch.bfloat16)
        seq_ops.attn_ragged(q, kp, vp, None, out, b, H, G, dim, vdim, dim ** -0.5, 0.0, size, decode_kernel=False)
        outs.append(out)
    assert outs[0].isfinite().all() and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("window,keep", [(None, 0), (70, 3)])
@pytest.mark.parametrize("n,ctx", [(5, 60), (64, 0), (130, 131)])
def test_what_no_row_sees_stays_out(softcap, window, keep, n, ctx):
    """Rows past the last key of a sequence hold anything (pages are reused); keys that leave the window and scores of +-10^4 take part as the masks and the maximum say."""
    H, G, dim = 4, 2, 64
    q = 100 * torch.randn(n, H * dim, device="cuda").bfloat16()
    k = torch.full((384, G * dim), float("nan"), device="cuda", dtype=torch.bfloat16)
    v = k.clone()
    k[:n + ctx], v[:n + ctx] = 100 * torch.randn(n + ctx, G * dim, device="cuda"), torch.randn(n + ctx, G * dim, device="cuda")
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=ctx, slot=0, pages=list(range(6)))])
    b.page_table, b.max_pages, b.singles = torch.arange(6, device="cuda", dtype=torch.int32).view(1, -1).contiguous(), 6, 0
    out = torch.empty(n, H * dim, device="cuda", dtype=torch.bfloat16)
    score = None if window is None else seq_ops.ScoreOptions(H, window=window, keep_first=keep)
    seq_ops.attn_ragged(q, k.view(6, 64, -1), v.view(6, 64, -1), None, out, b, H, G, dim, dim, dim ** -0.5, softcap, 64, decode_kernel=False, score=score)
    qd, kd, vd = (t.double() for t in (q.view(n, H, dim), k[:n + ctx].view(-1, G, dim).repeat_interleave(H // G, 1), v[:n + ctx].view(-1, G, dim).repeat_interleave(H // G, 1)))
    s = torch.einsum("qhd,khd->hqk", qd, kd) * dim ** -0.5
    s = softcap * torch.tanh(s / softcap) if softcap else s
    away = (ctx + torch.arange(n, device="cuda"))[:, None] - torch.arange(n + ctx, device="cuda")[None]
    seen = (away >= 0) & ((away < (window or 10 ** 9)) | (torch.arange(n + ctx, device="cuda")[None] < keep))
    want = torch.einsum("hqk,khd->qhd", s.masked_fill(~seen, -float("inf")).softmax(-1), vd).reshape(n, -1)
    # a score is 64 products of about 10^4 added up in fp32 and divided by 8: its error stays below 64 2^-24 64 10^4 / 8 = 0.3, so rows whose two best scores are
    # more than 12 apart are their best key's value; capped scores saturate at +-30, and where they do not the score and its error are a thousandth of that
    assert out.isfinite().all()
    near = (s.masked_fill(~seen, -float("inf")).topk(2, -1).values.diff(dim=-1).abs() > 12).squeeze(-1).T if not softcap and n + ctx > 1 else None
    got = out.double().view(n, H, dim)
    ok = ((got - want.view(n, H, dim)).abs() <= 2.0 ** -7 * vd.abs().max()).all(-1)
    assert ok.all() if near is None else ok[near].all()
