"""Kernels of a decode step on the ragged engine where their vector forms can go wrong (edges of tiles, remainders, smallest sizes), against 64-bit sums.

Bounds: fp32 results of sums of n products lie within a few n^(1/2) 2^-24 of the largest term's scale (1e-5 here); bf16 outputs within one rounding (2^-8 of the
value, 2^-9 of it on average)."""
import math

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu
DT = [torch.bfloat16, torch.float32]


def _t(*shape, seed=0, dtype=torch.float32, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _close(got, want, dtype, scale=None):
    got, want = got.double(), want.double()
    s = want.abs().max().item() if scale is None else scale
    tol = want.abs() * 2.0 ** -8 + 1e-5 * s if dtype == torch.bfloat16 else torch.full_like(want, 1e-5 * s)
    assert ((got - want).abs() <= tol).all(), ((got - want).abs() - tol).max().item()


def _decode_batch(ctxs, page=64):
    rows, first = [], 0
    for i, c in enumerate(ctxs):
        n = c // page + 1
        rows.append(dict(tokens=[1], ctx=c, slot=i, pages=list(range(first, first + n))))
        first += n
    return seq_ops.make_step_batch(rows), first


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("G,gsz,dim,vdim", [(2, 4, 64, 64), (1, 1, 8, 8), (2, 9, 72, 64), (1, 5, 128, 128), (3, 2, 40, 104), (1, 4, 200, 16)])
@pytest.mark.parametrize("window,keep", [(0, 0), (33, 0), (40, 5)])
def test_single_token_attention(dtype, G, gsz, dim, vdim, window, keep):
    ctxs = [0, 1, 30, 31, 32, 63, 64, 127, 300, 1100]
    H = G * gsz
    b, pages = _decode_batch(ctxs)
    q, kp, vp = _t(b.T, H * dim, seed=1, dtype=dtype), _t(pages, 64, G * dim, seed=2, dtype=dtype), _t(pages, 64, G * vdim, seed=3, dtype=dtype)
    last = b.page_table.cpu()
    for e, c in enumerate(ctxs):  # rows behind the newest token are what earlier owners of the page left
        kp[last[e, c // 64], c % 64 + 1:] = float("nan")
        vp[last[e, c // 64], c % 64 + 1:] = float("nan")
    out = torch.empty(b.T, H * vdim, device="cuda", dtype=dtype)
    score = seq_ops.ScoreOptions(H, window or None, keep)
    seq_ops.attn_ragged(q, kp, vp, None, out, b, H, G, dim, vdim, dim ** -0.5, 0.0, 64, score=score)
    for e, c in enumerate(ctxs):
        rows = last[e, : c // 64 + 1].tolist()
        k = torch.cat([kp[p] for p in rows])[: c + 1].double().view(c + 1, G, dim)
        v = torch.cat([vp[p] for p in rows])[: c + 1].double().view(c + 1, G, vdim)
        s = torch.einsum("gid,jgd->gij", q[e].double().view(G, gsz, dim), k) * dim ** -0.5
        j = torch.arange(c + 1, device="cuda")
        if window:
            s = s.masked_fill(~((c - j < window) | (j < keep)), -math.inf)
        want = torch.einsum("gij,jgd->gid", torch.softmax(s, -1), v).reshape(-1)
        _close(out[e], want, dtype, scale=max(1.0, v.abs().max().item()))


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("H,dim,vdim", [(3, 64, 64), (1, 128, 128), (2, 20, 68), (2, 7, 4), (1, 100, 132)])
def test_recurrent_scan(dtype, H, dim, vdim):
    ns, ctxs = [1, 3, 1, 2], [5, 0, 0, 9]
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=c, slot=s, pages=[s]) for n, c, s in zip(ns, ctxs, [2, 0, 3, 1])])
    qkv = _t(b.T, H * (2 * dim + vdim), seed=4, dtype=dtype)
    state = _t(5, H, dim, vdim, seed=5)
    want_state, decay = state.double().clone(), torch.linspace(0.7, 0.99, H, device="cuda")
    out = torch.empty(b.T, H * vdim, device="cuda")
    L = _lib.lib()
    _lib.check(L.pg_linear_attn_scan(qkv.data_ptr(), qkv.stride(0), state.data_ptr(), decay.data_ptr(), out.data_ptr(), b.row0.data_ptr(), b.n.data_ptr(),
                                     b.ctx.data_ptr(), b.slot.data_ptr(), b.E, H, dim, vdim, 0, int(dtype == torch.float32), _lib.stream()), "scan")
    r = 0
    for n, c, s in zip(ns, ctxs, [2, 0, 3, 1]):
        S = want_state[s] if c else torch.zeros_like(want_state[s])
        for _ in range(n):
            x = torch.nn.functional.silu(qkv[r].double())
            q, k, v = x[: H * dim].view(H, dim), x[H * dim: 2 * H * dim].view(H, dim), x[2 * H * dim:].view(H, vdim)
            S = decay.double()[:, None, None] * S + k[:, :, None] * v[:, None, :]
            _close(out[r], torch.einsum("hdv,hd->hv", S, q).reshape(-1), torch.float32, scale=10.0)
            r += 1
        want_state[s] = S
    _close(state, want_state, torch.float32, scale=10.0)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("H,dim,vdim", [(2, 64, 64), (1, 128, 128), (2, 20, 68), (1, 7, 4)])
@pytest.mark.parametrize("turned", [False, True])
def test_recurrent_scan_of_long_portions(dtype, H, dim, vdim, turned):
    """Token by token where blocks are the rule: every token's q, k and v are requested a token ahead."""
    ns, ctxs = [33, 1, 70], [4, 0, 0]
    b = seq_ops.make_step_batch([dict(tokens=[1] * n, ctx=c, slot=s, pages=[2 * s, 2 * s + 1]) for n, c, s in zip(ns, ctxs, [2, 0, 1])])
    qkv, state = _t(b.T, H * (2 * dim + vdim), seed=4, dtype=dtype), _t(3, H, dim, vdim, seed=5)
    want_state, decay, out = state.double().clone(), torch.linspace(0.7, 0.95, H, device="cuda"), torch.empty(b.T, H * vdim, device="cuda")
    angles = torch.linspace(0, 3, b.T, device="cuda", dtype=torch.float64)[:, None] * torch.linspace(1, 0.1, (dim + 7) // 8 * 4, device="cuda", dtype=torch.float64)
    table = torch.stack([angles.cos(), angles.sin()], 1).float().contiguous() if turned else None
    if turned:
        seq_ops.retention(qkv, state, decay, out, b, H, dim, vdim, kscale=0.5, rotate=table, blocks=False)
    else:
        seq_ops.linear_attn(qkv, state, decay, out, b, H, dim, vdim, chunked=False)

    def turn(x, t):
        y = x.clone()
        for i in range(dim // 2):
            c, s = table[t, 0, i].double(), table[t, 1, i].double()
            y[:, 2 * i], y[:, 2 * i + 1] = x[:, 2 * i] * c - x[:, 2 * i + 1] * s, x[:, 2 * i + 1] * c + x[:, 2 * i] * s
        if dim % 2:  # the last element has no partner (its pair's other half is zero)
            y[:, dim - 1] = x[:, dim - 1] * table[t, 0, dim // 2].double()
        return y

    r = 0
    for n, c, slot in zip(ns, ctxs, [2, 0, 1]):
        S = want_state[slot] if c else torch.zeros_like(want_state[slot])
        for _ in range(n):
            x = qkv[r].double() if turned else torch.nn.functional.silu(qkv[r].double())
            q, k, v = x[: H * dim].view(H, dim), x[H * dim: 2 * H * dim].view(H, dim), x[2 * H * dim:].view(H, vdim)
            if turned:
                q, k = turn(q, r), turn(k, r) * 0.5
            S = decay.double()[:, None, None] * S + k[:, :, None] * v[:, None, :]
            _close(out[r], torch.einsum("hdv,hd->hv", S, q).reshape(-1), torch.float32, scale=20.0)
            r += 1
        want_state[slot] = S
    _close(state, want_state, torch.float32, scale=20.0)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("D,groups", [(128, 1), (1024, 8), (1152, 3), (2048, 4), (4096, 1), (3968, 31)])
def test_norms_that_keep_their_row(dtype, D, groups):
    rows, eps = 5, 1e-5
    y, w, x = _t(rows, D, seed=6), _t(D, seed=7), _t(rows, D, seed=8)
    yd = y.double().view(rows, groups, -1)
    bare = (yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + eps)).view(rows, D) * w.double()
    want = x.double() + bare
    act = torch.empty(rows, D, device="cuda", dtype=dtype)
    seq_ops.group_rmsnorm_add(y, w, x, act, groups, eps)
    _close(x, want, torch.float32)
    _close(act, want, dtype)
    seq_ops.group_rmsnorm_add(y, w, None, act, groups, eps)
    _close(act, bare, dtype)
    both = _t(rows, 2 * D, seed=9, dtype=dtype)
    gate = both[:, D:]
    seq_ops.rmsnorm_gate(y, w, gate, act, eps)
    yd = y.double()
    _close(act, yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + eps) * w.double() * torch.sigmoid(gate.double()), dtype)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("D,col0,ld", [(8, 0, 8), (2048, 64, 2200), (4104, 8, 4112), (20, 4, 32)])
def test_embedding_rows(dtype, D, col0, ld):
    table = _t(50, ld, seed=10, dtype=dtype)
    tokens = torch.tensor([0, 49, 7], device="cuda", dtype=torch.int32)
    act = torch.empty(3, D, device="cuda", dtype=dtype)
    out = seq_ops.embed_rows(tokens, table, col0, D, 1.7, out_act=act)
    want = table[tokens.long(), col0: col0 + D].float() * 1.7
    assert torch.equal(out, want) and torch.equal(act, want.to(dtype))


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("rows,D,n,n_pad", [(1, 256, 1, 8), (5, 2048, 64, 64), (48, 1024, 60, 64), (3, 4096, 130, 136), (2, 8192, 256, 256), (128, 512, 7, 8)])
def test_side_input(dtype, rows, D, n, n_pad):
    eps = 1e-6
    g, p = torch.zeros(n_pad, D, device="cuda", dtype=dtype), torch.zeros(D, n_pad, device="cuda", dtype=dtype)
    g[:n], p[:, :n] = _t(n, D, seed=11, dtype=dtype, scale=D ** -0.5), _t(D, n, seed=12, dtype=dtype, scale=n ** -0.5)
    table, w, x = _t(20, 3 * n, seed=13, dtype=dtype), _t(D, seed=14), _t(rows, D, seed=15)
    tokens = torch.arange(rows, device="cuda", dtype=torch.int32) % 20
    act = x if dtype == torch.float32 else x.to(dtype)
    gz = torch.nn.functional.gelu(act.double() @ g[:n].double().T, approximate="tanh") * table[tokens.long(), n: 2 * n].double()
    seen = x.clone()
    seq_ops.token_side(act, g, tokens, table, n, n, p, w, x, None if dtype == torch.float32 else act, eps)
    # bf16: the inner values are rounded once, 2^-9 each, and the projection averages over n of them
    y = gz @ p[:, :n].double().T
    want = seen.double() + y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps) * w.double()
    tol = 2e-5 if dtype == torch.float32 else 2.0 ** -8
    assert ((x.double() - want).abs() <= tol * (1 + want.abs() + w.abs() * 4)).all()
    if dtype == torch.bfloat16:
        assert torch.equal(act, x.to(dtype))
