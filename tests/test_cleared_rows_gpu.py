"""A norm that leaves zeros where it read, and a product that sums into them: the register form (groups of whole 128), the others, row pitches, and sizes that share K out and that do not."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 48, 130])
@pytest.mark.parametrize("D,groups", [(2048, 4), (1024, 8), (640, 5), (96, 3), (30, 2), (5120, 1)])
@pytest.mark.parametrize("pitch", [0, 4])
def test_the_norm_is_the_same_and_its_input_zero(T, D, groups, pitch):
    g = torch.Generator(device="cuda").manual_seed(D)
    y = torch.randn(T, D + pitch, generator=g, device="cuda")
    x, w = torch.randn(T, D, generator=g, device="cuda"), torch.randn(D, generator=g, device="cuda")
    res = []
    for clear in (False, True):
        yy, xx, out = y.clone(), x.clone(), torch.empty(T, D, device="cuda", dtype=torch.bfloat16)
        seq_ops.group_rmsnorm_add(yy[:, :D], w, xx, out, groups, 1e-6, clear=clear)
        res.append((xx, out))
        assert torch.equal(yy[:, D:], y[:, D:]) and (not yy[:, :D].any() if clear else torch.equal(yy, y))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("T,F,K", [(1, 2048, 8192), (48, 2048, 8192), (48, 2048, 512), (128, 1024, 4096), (300, 1024, 4096), (5, 96, 1024)])
def test_the_product_is_the_same(T, F, K):
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(T, K, generator=g, device="cuda").to(torch.bfloat16), torch.randn(F, K, generator=g, device="cuda").to(torch.bfloat16)
    a = seq_ops.linear(x, w, torch.full((T, F), float("nan"), device="cuda"))
    b = seq_ops.linear(x, w, torch.zeros(T, F, device="cuda"), zeros=True)
    # the same products, parts of K added in any order: up to 2^-20 of the sum of magnitudes
    assert ((a - b).abs() <= 2.0 ** -20 * (x.abs().float() @ w.abs().float().T)).all()
