"""The vector forms of pg_attn_prepare, pg_latent_gather and pg_latent_pack_kv (whole 16-byte pieces) against the element-wise ones, which the same
calls take when a row starts off a 16-byte boundary."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


def _batch(entries):
    pages, rows = 0, []
    for n, ctx in entries:
        k = (n + ctx + 63) // 64
        rows.append(dict(tokens=[1] * n, ctx=ctx, slot=0, pages=list(range(pages, pages + k))))
        pages += k
    return seq_ops.make_step_batch(rows), pages


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("entries", [[(1, 70)] * 5, [(130, 0), (1, 3), (77, 60)], [(2500, 0)], [(2501, 0)], [(2400, 3), (103, 0)]])
@pytest.mark.parametrize("H,G,dim,vdim,rot", [(4, 2, 64, 64, 64), (6, 3, 16, 8, 6), (2, 1, 256, 32, 0), (8, 8, 32, 128, 10), (8, 1, 64, 64, 16)])
@pytest.mark.parametrize("norm_qk,norm_v,form", [(False, False, ""), (True, True, ""), (True, False, "keys"), (seq_ops.NORM_PROJECTION, False, "blend"), (seq_ops.NORM_PROJECTION, True, ""),
                                              (True, False, "queries")])
def test_attn_prepare(dtype, entries, H, G, dim, vdim, rot, norm_qk, norm_v, form):
    if norm_v or form == "keys":
        vdim = dim
    b, pages = _batch(entries)
    W = (H + G) * dim + (0 if form == "keys" else G * vdim)
    proj = torch.randn(b.T, W, device="cuda").to(dtype)
    freq = (10000.0 ** (-torch.arange(0, max(rot, 2), 2, dtype=torch.float64) / max(rot, 2))).cuda()
    sizes = (H * dim, G * dim) if norm_qk is seq_ops.NORM_PROJECTION else (dim, dim)
    qn, kn = (1 + 0.1 * torch.randn(n, device="cuda") for n in sizes)
    other = torch.randn(b.T, G * vdim, device="cuda").to(dtype) if form == "blend" else None
    outs = []
    for shift in (0, 1):  # a row pitch that is no multiple of 8 elements: the element-wise form
        x = torch.zeros(b.T, W + 8 + shift, device="cuda", dtype=dtype)[:, :W]
        x.copy_(proj)
        q = torch.full((b.T, H * dim), float("nan"), device="cuda", dtype=dtype)
        k, v = (torch.full((pages, 64, G * n), 7.0, device="cuda", dtype=dtype) for n in (dim, vdim))
        own = form != "queries"
        seq_ops.attn_prepare(x, b, freq, qn, kn, q, k if own else None, v if own else None, H, G, dim, vdim, rot, 1e-5, 64, norm_qk=norm_qk, norm_v=norm_v,
                             v_from_k=form == "keys", rot_gain=1.25, v_other=other, v_mix=0.3 if form == "blend" else 0.0)
        outs.append((q, k, v))
    # sums of squares in another order change a norm by up to 2^-20 of itself, and a rotated element is the difference of two products of
    # values up to 8 (6.3 before the gain of 1.25): |difference| <= 2^-20 * 16 before the rounding to the activation type, whatever cancels
    tol = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -19
    for a, c in zip(*outs):
        assert a.isfinite().all()
        assert ((a.double() - c.double()).abs() <= tol * c.double().abs() + 2.0 ** -16).all()
        assert torch.equal(a == 7.0, c == 7.0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,dim,rot,vdim,rank", [(3, 64, 32, 64, 256), (5, 16, 8, 24, 40), (2, 12, 6, 10, 20), (4, 64, 0, 64, 64)])
def test_latent_rows(dtype, H, dim, rot, vdim, rank):
    entries = [(70, 100), (1, 200), (3, 0), (129, 64)]
    b, pages = _batch(entries)
    cache = torch.randn(pages, 64, rank + rot, device="cuda").to(dtype)
    w = (torch.randn(H * (dim + vdim), rank, device="cuda") * rank ** -0.5).to(dtype)
    k, v = seq_ops.latent_expand(cache, b, w, H, dim, rot, vdim, rank, 64, seq_ops.Precision(dtype))
    page = 0
    for e, (n, ctx) in enumerate(entries):
        count, rows = (n + ctx + 63) // 64, cache[page:page + (n + ctx + 63) // 64].reshape(-1, rank + rot)[:n + ctx]
        page += count
        if n == 1:
            continue
        at = int(b.dense_row0[e])
        up = rows[:, :rank].double() @ w.double().T
        ks, vs = k[at:at + n + ctx].view(-1, H, dim + rot), v[at:at + n + ctx].view(-1, H, vdim)
        tol = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -18
        assert torch.equal(ks[:, :, dim:], rows[:, None, rank:].expand(-1, H, -1))
        assert (ks[:, :, :dim].double() - up[:, :H * dim].view(-1, H, dim)).abs().max() <= tol * up.abs().max()
        assert (vs.double() - up[:, H * dim:].view(-1, H, vdim)).abs().max() <= tol * up.abs().max()


@pytest.mark.parametrize("at", [0, 255, 256, 300])
def test_latent_rows_of_one_entry_among_many(at):
    H, dim, rot, vdim, rank = 3, 16, 8, 16, 32
    entries = [(1, 5)] * 310
    entries[at], entries[(at + 7) % 310] = (70, 30), (2, 0)
    b, pages = _batch(entries)
    cache = torch.randn(pages, 64, rank + rot, device="cuda").to(torch.bfloat16)
    w = (torch.randn(H * (dim + vdim), rank, device="cuda") * rank ** -0.5).to(torch.bfloat16)
    k, v = seq_ops.latent_expand(cache, b, w, H, dim, rot, vdim, rank, 64, seq_ops.Precision(torch.bfloat16))
    for e, (n, ctx) in enumerate(entries):
        if n == 1:
            continue
        first = int(b.page_table[e, 0])
        rows = cache[first:first + (n + ctx + 63) // 64].reshape(-1, rank + rot)[:n + ctx]
        at = int(b.dense_row0[e])
        up = rows[:, :rank].double() @ w.double().T
        ks, vs = k[at:at + n + ctx].view(-1, H, dim + rot), v[at:at + n + ctx].view(-1, H, vdim)
        assert torch.equal(ks[:, :, dim:], rows[:, None, rank:].expand(-1, H, -1))
        assert (ks[:, :, :dim].double() - up[:, :H * dim].view(-1, H, dim)).abs().max() <= 2.0 ** -7 * up.abs().max()
        assert (vs.double() - up[:, H * dim:].view(-1, H, vdim)).abs().max() <= 2.0 ** -7 * up.abs().max()
