"""The merge of a row's key splits: one and two columns a thread, widths past a CTA's threads, up to and past the 16 splits that are requested ahead, splits without keys; in 64 bits."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vdim", [1, 24, 63, 64, 130, 256, 257, 600])
@pytest.mark.parametrize("nsplit", [2, 15, 16, 17, 64])
def test_merge(dtype, vdim, nsplit):
    E, H = 3, 2
    g = torch.Generator(device="cuda").manual_seed(vdim)
    part = torch.randn(E, H, nsplit, vdim + 2, generator=g, device="cuda")
    part[..., 1] = part[..., 1].abs() + 0.5
    part[:, :, 1::3, 0], part[:, :, 1::3, 1:] = -float("inf"), float("nan")  # splits that saw no key
    gate = torch.randn(E, H, generator=g, device="cuda").to(dtype)
    row0, n = torch.arange(E, device="cuda", dtype=torch.int32), torch.tensor([1, 2, 1], device="cuda", dtype=torch.int32)
    out = torch.full((E, H, vdim), 7.0, device="cuda", dtype=dtype)
    _lib.check(_lib.lib().pg_attn_decode_merge(part.data_ptr(), gate.data_ptr(), H, out.data_ptr(), row0.data_ptr(), n.data_ptr(), E, nsplit, H, vdim, 1, int(dtype == torch.float32), 0,
                                               _lib.stream()), "pg_attn_decode_merge")
    seen = part[..., 0].isfinite()
    f = torch.where(seen, torch.exp(part[..., 0].double() - part[..., 0].double().amax(-1, keepdim=True)), 0.0)
    p = torch.where(seen[..., None], part.double(), 0.0)
    want = (f[..., None] * p[..., 2:]).sum(2) / (f * p[..., 1]).sum(-1)[..., None] * torch.sigmoid(gate.double())[..., None]
    # up to 64 fp32 terms and expf: 2^-19 of the sum of magnitudes; one rounding to the activation type
    scale = (f[..., None] * p[..., 2:].abs()).sum(2) / (f * p[..., 1]).sum(-1)[..., None]
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20) * want.abs() + 2.0 ** -19 * scale
    assert (out[1] == 7).all() and ((out.double() - want).abs() <= tol)[[0, 2]].all()


@pytest.mark.parametrize("dim,vdim", [(96, 64), (288, 256), (544, 512)])
@pytest.mark.parametrize("H", [3, 32, 70])
def test_splits_of_latent_rows_in_scratch_off_eight_bytes(dim, vdim, H):
    """The splits of pg_attn_latent_decode_mma and their merge take scratch that starts on any float: the same bits as on sixteen bytes."""
    E, ctx, nsplit = 3, 700, 5
    g = torch.Generator(device="cuda").manual_seed(dim)
    q = torch.randn(E, H, dim, generator=g, device="cuda").to(torch.bfloat16)
    pages = torch.randn(11, 64, dim, generator=g, device="cuda").to(torch.bfloat16)
    row0, n, ctxs = torch.arange(E, device="cuda", dtype=torch.int32), torch.ones(E, device="cuda", dtype=torch.int32), torch.tensor([ctx, 3, 130], device="cuda", dtype=torch.int32)
    table = torch.arange(11, device="cuda", dtype=torch.int32).repeat(E, 1)
    outs = []
    for shift in (0, 1):
        part = torch.full((E * H * nsplit * (vdim + 2) + 1,), float("nan"), device="cuda")[shift:]
        out = torch.full((E, H, vdim), 7.0, device="cuda", dtype=torch.bfloat16)
        L, st = _lib.lib(), _lib.stream()
        _lib.check(L.pg_attn_latent_decode_mma(q.data_ptr(), pages.data_ptr(), 0, 0, out.data_ptr(), part.data_ptr(), row0.data_ptr(), n.data_ptr(), ctxs.data_ptr(), table.data_ptr(), 11, 64,
                                               E, nsplit, H, dim, vdim, dim ** -0.5, 0, st), "pg_attn_latent_decode_mma")
        _lib.check(L.pg_attn_decode_merge(part.data_ptr(), 0, 0, out.data_ptr(), row0.data_ptr(), n.data_ptr(), E, nsplit, H, vdim, 1, 0, 0, st), "pg_attn_decode_merge")
        outs.append(out)
    assert torch.equal(*outs)
    k = pages.view(-1, dim)[:ctx + 1].double()
    want = torch.softmax(q[0].double() @ k.T * dim ** -0.5, -1) @ k[:, :vdim]
    # rows of standard normals: P carries 24 bits, the result one rounding to bf16
    assert ((outs[0][0].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all()
