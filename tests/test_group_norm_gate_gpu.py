"""Gated group norms whose lanes share a warp: group sizes from one lane to a whole warp of eight float4, one and two float4 a lane (few and many rows), against 64 bits."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("groups,gs", [(5, 4), (3, 8), (7, 32), (32, 64), (3, 128), (2, 512), (3, 1024), (4, 48)])
@pytest.mark.parametrize("cells", [3000, 1100000])
def test_sizes(dtype, groups, gs, cells):
    D = groups * gs
    rows = cells // D + 1
    g = torch.Generator(device="cuda").manual_seed(gs)
    o, z = torch.randn(rows, D, generator=g, device="cuda"), torch.randn(rows, D, generator=g, device="cuda").to(dtype)
    for w in (torch.randn(gs, generator=g, device="cuda"), torch.randn(D, generator=g, device="cuda"), None):
        for mode in (seq_ops.GATE_SIGMOID_AFTER, seq_ops.GATE_SILU_BEFORE, seq_ops.GATE_SILU_AFTER):
            out = torch.empty(rows, D, device="cuda", dtype=dtype)
            seq_ops.group_norm_gate(o, w, z, out, groups, 1e-5, mode, scale=0.7)
            x, zz = o.double(), z.double()
            if mode == seq_ops.GATE_SILU_BEFORE:
                x = x * zz * torch.sigmoid(zz)
            x = x.view(rows, groups, gs)
            x = 0.7 * x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
            if w is not None:
                x = x * w.double().view(-1, gs)
            x = x.reshape(rows, D)
            if mode != seq_ops.GATE_SILU_BEFORE:
                x = x * torch.sigmoid(zz) * (zz if mode == seq_ops.GATE_SILU_AFTER else 1)
            # fp32: sums and the exponential's argument (z log2 e, |z| < 6) to 2^-20; bf16: the hardware exponential (2^-19) far below the rounding by 2^-9
            tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
            assert ((out.double() - x).abs() <= tol * x.abs() + 2.0 ** -20).all()
