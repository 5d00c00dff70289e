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
