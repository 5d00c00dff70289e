"""Patch rows of images: patches per CTA that do not divide a row, odd patch sizes, pixels off 8 bytes, rows off 16 bytes and patches wider than the staging area; bytes equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,P,hp,wp,extra", [(2, 3, 14, 16, 16, 20), (1, 3, 14, 3, 5, 4), (3, 3, 16, 2, 7, 0), (2, 1, 7, 4, 9, 7), (1, 4, 1, 5, 3, 4), (1, 2, 2, 3, 33, 8), (1, 3, 64, 2, 3, 8),
                                              (2, 7, 64, 1, 2, 8)])
@pytest.mark.parametrize("shift_in,shift_out", [(0, 0), (1, 0), (0, 1), (0, 2)])
def test_rows(B, C, P, hp, wp, extra, shift_in, shift_out):
    from paligemma_multimodal_system_b200 import _lib
    H, W, K = hp * P, wp * P, C * P * P
    Kp = K + extra
    assert Kp % 8 == 0
    px = torch.randn(B * C * H * W + shift_in, device="cuda")[shift_in:].view(B, C, H, W)
    out = torch.full((B * hp * wp * Kp + shift_out + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    _lib.check(_lib.lib().pg_im2col(px.data_ptr(), out[shift_out:].data_ptr(), B, C, H, W, P, Kp, _lib.stream()), "pg_im2col")
    want = px.view(B, C, hp, P, wp, P).permute(0, 2, 4, 1, 3, 5).reshape(B * hp * wp, K).to(torch.bfloat16)
    got = out[shift_out:shift_out + B * hp * wp * Kp].view(-1, Kp)
    assert torch.equal(got[:, :K], want) and not got[:, K:].any()
    assert (out[:shift_out] == 7).all() and (out[shift_out + B * hp * wp * Kp:] == 7).all()
