"""Delta rule in blocks of 16 tokens where decays over a block leave the normal numbers: a factor below 2^-126 on a value of 2^100 is no zero."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 64)])
def test_strong_decay_of_a_large_value(dim, vdim):
    """Channel 0 takes 2^100 at the first token and decays by 2^-8.41 a token; every query reads it.  After fifteen of them 2^-26.2 is left of it."""
    n, rate = 24, 8.41
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=0, slot=0, pages=[0])])
    q, k, v = (torch.zeros(n, d, device="cuda", dtype=torch.bfloat16) for d in (dim, dim, vdim))
    q[:, 0], k[0, 0], k[1:, 1], v[0] = 1, 1, 1, 2.0 ** 100
    beta = torch.full((n, 1), 60.0, device="cuda", dtype=torch.bfloat16)  # sigmoid: 1
    z = torch.log(torch.expm1(torch.tensor(rate, dtype=torch.float64) * torch.log(torch.tensor(2.0, dtype=torch.float64)))).item()  # its softplus is rate * ln 2
    decay = torch.full((n, dim), z, device="cuda")
    state, out = torch.zeros(1, 1, dim, vdim, device="cuda"), torch.full((n, vdim), float("nan"), device="cuda")
    seq_ops.delta_rule(q, k, v, beta, torch.ones(n, 2, device="cuda"), decay, torch.zeros(1, device="cuda"), torch.zeros(dim, device="cuda"), state, out, b, 1, 1, dim, vdim, blocks=True)
    want = 2.0 ** (100 - rate * torch.arange(n, device="cuda", dtype=torch.float64))
    # a factor of 2^-126.2 enters the products in bf16 terms of which the smallest is 2^-133: 2^-7 of it; fp32 exponents to 2^-20
    assert ((out.double() - want[:, None]).abs() <= 2.0 ** -6 * want[:, None]).all()
    assert ((state[0, 0, 0].double() - want[-1]).abs() <= 2.0 ** -6 * want[-1]).all() and (state[0, 0, 2:] == 0).all()
