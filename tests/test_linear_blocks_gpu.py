"""Decayed linear attention with silu in blocks on the tensor cores: block remainders, head sizes of every build, few CTAs (two per SM) and many (three), continued and fresh slots, mixed
with single tokens, against 64 bits and no further from them than the token-by-token form."""
import pytest
import torch

from paligemma_multimodal_system_b200 import seq_ops

pytestmark = pytest.mark.gpu


def _case(ns, ctxs, H, dim, vdim, seed=1):
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=c, slot=i, pages=list(range((n + c + 63) // 64))) for i, (n, c) in enumerate(zip(ns, ctxs))])
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = torch.randn(b.T, H * (2 * dim + vdim), generator=g, device="cuda").to(torch.bfloat16)
    state = torch.randn(len(ns), H, dim, vdim, generator=g, device="cuda")
    decay = 1.0 - 2.0 ** (-4 - 3 * torch.arange(H, device="cuda") / H)
    return b, qkv, state, decay


def _want(qkv, state, decay, H, dim, vdim):
    n = qkv.shape[0]
    x = torch.nn.functional.silu(qkv.double())
    q, k, v = x[:, :H * dim].view(n, H, dim), x[:, H * dim:2 * H * dim].view(n, H, dim), x[:, 2 * H * dim:].view(n, H, vdim)
    S, a, out = state.double(), decay.double()[:, None, None], []
    for t in range(n):
        S = a * S + k[t][:, :, None] * v[t][:, None, :]
        out.append((S * q[t][:, :, None]).sum(1))
    return torch.stack(out).view(n, H * vdim), S


def _far(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("H,dim,vdim", [(64, 64, 64), (64, 32, 64), (32, 96, 72), (32, 128, 128), (64, 40, 24), (500, 64, 64)])
@pytest.mark.parametrize("ns,ctxs", [((8, 33), (0, 0)), ((31, 1, 32), (5, 70, 0)), ((65, 7), (64, 3)), ((200,), (9,))])
def test_blocks(H, dim, vdim, ns, ctxs):
    b, qkv, state, decay = _case(ns, ctxs, H, dim, vdim)
    res = []
    for chunked in (None, False):
        st, out = state.clone(), torch.full((b.T, H * vdim), float("nan"), device="cuda")
        seq_ops.linear_attn(qkv, st, decay, out, b, H, dim, vdim, chunked=chunked)
        res.append((out, st))
    r = 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        want, S = _want(qkv[r:r + n], state[i] * (c > 0), decay, H, dim, vdim)
        (o1, s1), (o2, s2) = ((x[r:r + n], y[i]) for x, y in res)
        # three bf16 terms keep 24 bits; a tensor product cuts its sum off below 2^-23 once per 16 of the depth, silu adds 2^-22: 2^-21 in all
        assert _far(o1, want) <= 2.0 ** -21 and _far(s1, S) <= 2.0 ** -21
        assert _far(o1, want) <= 1.25 * _far(o2, want) + 2.0 ** -25 and _far(s1, S) <= 1.25 * _far(s2, S) + 2.0 ** -25
        r += n


def test_a_value_that_is_not_finite_stays_with_its_column_and_the_tokens_of_its_sixteen():
    b, qkv, state, decay = _case((100,), (0,), 64, 64, 64)
    clean = torch.empty(b.T, 64 * 64, device="cuda")
    seq_ops.linear_attn(qkv, state.clone(), decay, clean, b, 64, 64, 64)
    qkv[50, 2 * 64 * 64 + 5] = float("inf")
    out = torch.empty_like(clean)
    seq_ops.linear_attn(qkv, state.clone(), decay, out, b, 64, 64, 64)
    other = torch.ones(64 * 64, dtype=torch.bool, device="cuda")
    other[5] = False
    assert torch.equal(out[:, other], clean[:, other]) and torch.equal(out[:48, 5], clean[:48, 5]) and not out[50:, 5].isfinite().any()


@pytest.mark.parametrize("H,dim,vdim", [(16, 64, 64), (3, 32, 72), (5, 128, 128)])
@pytest.mark.parametrize("ns", [(200,) + (1,) * 40, (1, 1, 70, 1, 7)])
def test_one_portion_among_single_tokens(H, dim, vdim, ns):
    """Single tokens own no blocks: a few heads of one portion take the FMA blocks in the widths of one entry, the others go token by token."""
    ctxs = [(13 * i) % 40 for i in range(len(ns))]
    b, qkv, state, decay = _case(ns, ctxs, H, dim, vdim)
    st, out = state.clone(), torch.full((b.T, H * vdim), float("nan"), device="cuda")
    seq_ops.linear_attn(qkv, st, decay, out, b, H, dim, vdim)
    r = 0
    for i, (n, c) in enumerate(zip(ns, ctxs)):
        want, S = _want(qkv[r:r + n], state[i] * (c > 0), decay, H, dim, vdim)
        # fp32 sums of up to 200 tokens and 128 products, silu to 2^-22: 2^-20
        assert _far(out[r:r + n], want) <= 2.0 ** -20 and _far(st[i], S) <= 2.0 ** -20
        r += n
