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
