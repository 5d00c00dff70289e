"""fp32 products as six bf16 products of three-term operands, at the edges of their tiles and of fp32.

Bound: a product of two values loses at most about 2^-23 of itself, a 64-deep partial sum a few 2^-24 of its size, and partial sums are added to nearest; 4e-7 of the
norm of the result leaves twice the largest error seen (1.5e-7), and is no more than what a chain of fp32 FMAs shows (2.9e-7 .. 5.8e-7)."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu


def _t(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda") * scale


def _split(x, w, out, bias=None, accumulate=0, scale=1.0, slack=0):
    (T, K), F = x.shape, w.shape[0]
    need = 16 + 6 * (T + F) * K + 4 * 16 * T * F
    scratch = torch.full((need + slack,), 0xFF, device="cuda", dtype=torch.uint8)  # (NaNs, and a raised flag)
    rc = _lib.lib().pg_gemm_fp32_split(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), _lib.ptr(bias), accumulate, scale, T, F, K,
                                       scratch.data_ptr(), need, _lib.stream())
    return rc


@pytest.mark.parametrize("T,F,K", [(1, 4, 8), (32, 64, 64), (127, 252, 72), (129, 260, 136), (255, 256, 1032), (256, 1024, 64), (257, 516, 8200), (700, 2048, 200), (33, 20000, 128)])
@pytest.mark.parametrize("full", [False, True])
def test_against_64_bits(T, F, K, full):
    """full: operands and output are views of wider tensors, with bias, scale and an output that is added to."""
    pad = 4 if full else 0
    x, w = _t(T, K + pad, seed=1)[:, :K], _t(F, K + 2 * pad, seed=2, scale=K ** -0.5)[:, :K]
    whole = _t(T, F + pad, seed=3)
    out, before = whole[:, :F], whole.clone()
    bias = _t(F, seed=4) if full else None
    want = x.double() @ w.double().T
    if full:
        want = (want + bias.double()) * 0.7 + out.double()
    assert _split(x, w, out, bias, int(full), 0.7 if full else 1.0) == 0
    assert ((out.double() - want).norm() / want.norm()).item() < 4e-7
    if pad:
        assert torch.equal(whole[:, F:], before[:, F:])


def test_no_further_from_64_bits_than_fmas():
    for seed, (T, F, K) in enumerate([(300, 512, 2048), (150, 300, 8192), (700, 256, 1024)]):
        x, w = _t(T, K, seed=10 + seed), _t(F, K, seed=20 + seed, scale=K ** -0.5)
        a, b = torch.empty(T, F, device="cuda"), torch.empty(T, F, device="cuda")
        assert _split(x, w, a) == 0
        _lib.check(_lib.lib().pg_gemm_simt(x.data_ptr(), K, w.data_ptr(), K, b.data_ptr(), F, T, F, K, 1, 1, _lib.stream()), "simt")
        want = x.double() @ w.double().T
        assert (a.double() - want).norm() <= (b.double() - want).norm()


@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["x", "w"])
def test_infinities_and_nans_are_those_of_the_plain_products(bad, where):
    T, F, K = 300, 260, 136
    x, w = _t(T, K, seed=5).to(torch.bfloat16).float(), _t(F, K, seed=6).to(torch.bfloat16).float()  # (second and third terms zero: inf * 0 if it were split)
    (x if where == "x" else w)[7, 130] = bad
    a, b, bias = _t(T, F, seed=7), _t(T, F, seed=7), _t(F, seed=8)
    assert _split(x, w, a, bias, 1, 0.5) == 0
    _lib.check(_lib.lib().pg_gemm_simt_bias(x.data_ptr(), K, w.data_ptr(), K, b.data_ptr(), F, bias.data_ptr(), 1, 0.5, T, F, K, 1, 1, _lib.stream()), "simt")
    assert torch.equal(a, b) or torch.equal(torch.nan_to_num(a, 3.25), torch.nan_to_num(b, 3.25))
    assert not torch.isfinite(a).all()


def test_range_of_fp32():
    T, F, K = 64, 64, 64
    big = torch.tensor(3.4028234e38, device="cuda")
    x, w = torch.zeros(T, K, device="cuda"), torch.zeros(F, K, device="cuda")
    x[:, 0], w[:, 0] = big, 1.0          # rounds to infinity in bf16
    x[:, 1], w[:, 1] = 1e-30, 1e-30      # underflows
    out = torch.empty(T, F, device="cuda")
    assert _split(x, w, out) == 0
    assert torch.isfinite(out).all() and ((out - big).abs() <= 2 ** -22 * big).all()
    x[:, 0], w[:, 0] = 2e-36, 0.75       # third terms are below the normal numbers
    x[:, 1] = 0
    assert _split(x, w, out) == 0
    assert ((out.double() - 1.5e-36).abs() <= 2 ** -16 * 1.5e-36).all()


@pytest.mark.parametrize("K", [64, 1000])
@pytest.mark.parametrize("xs,ws", [(1e30, 1e30), (3e38, 3e38), (2.5e18, 7e19), (1e-10, 3.3e38), (1.0, 3.4e38)])
def test_products_at_the_end_of_the_range(xs, ws, K):
    """Finite operands, products near or above the largest fp32 and with all three terms: infinities where plain FMAs have infinities, never a NaN in their place."""
    T, F = 300, 260
    x, w = _t(T, K, seed=31).sign() * (1 + 0.1 * _t(T, K, seed=32).clamp(-1, 0)) * xs, _t(F, K, seed=33).abs().clamp(0.9, 1) * ws
    x[:100] = x[:100].abs()  # rows whose sums overflow to one side only
    assert torch.isfinite(x).all() and torch.isfinite(w).all()
    a, b = torch.empty(T, F, device="cuda"), torch.empty(T, F, device="cuda")
    assert _split(x, w, a) == 0
    _lib.check(_lib.lib().pg_gemm_simt(x.data_ptr(), K, w.data_ptr(), K, b.data_ptr(), F, T, F, K, 1, 1, _lib.stream()), "simt")
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
    ok = torch.isfinite(b)
    assert torch.equal(a[~ok & ~b.isnan()], b[~ok & ~b.isnan()])
    # finite sums: either is within K 2^-24 of the sum of the terms' sizes
    size = (x.double().abs() @ w.double().abs().T)[ok]
    assert ((a.double()[ok] - b.double()[ok]).abs() <= size * (2.0 ** -23 * K)).all()


@pytest.mark.parametrize("ex,ew,K,split", [(59, 59, 64, True), (60, 3, 64, False), (-100, 60, 64, False), (57, 57, 1000, True), (57, 57, 1024, True), (58, 0, 1024, False), (-120, 56, 1032, True), (57, -3, 1032, False),
                                           (63, 62, 64, False), (-110, 126, 64, False)])
def test_the_line_to_the_plain_products(ex, ew, K, split):
    """Operands of 1.5 x 2^e: split while e of each is at most (124 - log2 K) / 2 (then 2^(e_x + e_w + 2) K is at most 2^126), and the sums are right on either side."""
    T, F = 64, 64
    x, w = torch.full((T, K), 1.5 * 2.0 ** ex, device="cuda"), torch.full((F, K), 1.5 * 2.0 ** ew, device="cuda")
    scratch = torch.zeros(1 << 22, device="cuda", dtype=torch.uint8)
    out = torch.empty(T, F, device="cuda")
    assert _lib.lib().pg_gemm_fp32_split(x.data_ptr(), K, w.data_ptr(), K, out.data_ptr(), F, 0, 0, 1.0, T, F, K, scratch.data_ptr(), scratch.numel(), _lib.stream()) == 0
    assert scratch[:4].view(torch.int32).item() == int(not split)
    want = (x.double() @ w.double().T).float()
    assert torch.equal(out.isinf(), want.isinf()) and torch.allclose(out, want, rtol=1e-6)


@pytest.mark.parametrize("T,F,K", [(300, 40000, 2048), (30000, 260, 2048), (11000, 11004, 4096), (300, 22020, 2048), (300, 4100, 16384)])
def test_large_operands_in_blocks(T, F, K):
    """More than 256 MB of planes: blocks of features, of tokens, of both; the last block short.  Views, bias, scale, an output that is added to."""
    L = _lib.lib()
    need = L.pg_gemm_fp32_scratch(T, F, K)
    assert 0 < need <= 256 << 20 < 6 * (T + F) * K
    x, w, bias = _t(T, K + 4, seed=41)[:, :K], _t(F, K, seed=42, scale=K ** -0.5), _t(F, seed=43)
    whole = _t(T, F + 4, seed=44)
    out, before = whole[:, :F], whole.clone()
    scratch = torch.full((need + 64,), 0xFF, device="cuda", dtype=torch.uint8)
    assert L.pg_gemm_fp32_split(x.data_ptr(), x.stride(0), w.data_ptr(), K, out.data_ptr(), out.stride(0), bias.data_ptr(), 1, 0.7, T, F, K, scratch.data_ptr(), need,
                                _lib.stream()) == 0
    assert (scratch[need:] == 0xFF).all() and torch.equal(whole[:, F:], before[:, F:])
    xd = x.double()
    for f in range(0, F, 4096):
        want = (xd @ w[f:f + 4096].double().T + bias[f:f + 4096].double()) * 0.7 + before[:, f:min(F, f + 4096)].double()
        assert ((out[:, f:f + 4096].double() - want).norm() / want.norm()).item() < 4e-7
    assert L.pg_gemm_fp32_split(x.data_ptr(), x.stride(0), w.data_ptr(), K, out.data_ptr(), out.stride(0), 0, 0, 1.0, T, F, K, scratch.data_ptr(), need - 1, _lib.stream()) != 0


def test_scratch_is_bounded():
    L = _lib.lib()
    for T in (32, 100, 750, 5000, 100000):
        for F, K in ((257216, 2048), (16384, 2048), (2048, 16384), (64, 64), (1 << 20, 8192), (256, 1 << 20)):
            assert 0 <= L.pg_gemm_fp32_scratch(T, F, K) <= 256 << 20
    assert L.pg_gemm_fp32_scratch(750, 16384, 2048) == 16 + 6 * (750 + 16384) * 2048  # (one block)


def test_no_room_for_the_scratch(monkeypatch):
    """A device without memory for the planes: the plain FMAs, with the bits they have."""
    K = 2048
    x, w = _t(700, K, seed=51), _t(K, K, seed=52)
    assert _lib.lib().pg_gemm_fp32_scratch(700, K, K) > 0
    real, out, acc = torch.empty, torch.empty(700, K, device="cuda"), _t(700, K, seed=53)

    def full(*a, dtype=None, **kw):
        if dtype == torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return real(*a, dtype=dtype, **kw)

    want = torch.empty(700, K, device="cuda")
    _lib.check(_lib.lib().pg_gemm_simt(x.data_ptr(), K, w.data_ptr(), K, want.data_ptr(), K, 700, K, K, 1, 1, _lib.stream()), "simt")
    want_acc = acc.clone()
    _lib.check(_lib.lib().pg_gemm_simt_bias(x.data_ptr(), K, w.data_ptr(), K, want_acc.data_ptr(), K, 0, 1, 0.5, 700, K, K, 1, 1, _lib.stream()), "simt")
    monkeypatch.setattr(seq_ops.torch, "empty", full)
    assert torch.equal(seq_ops.linear(x, w, out), want)
    assert torch.equal(seq_ops.linear_add(x, w, acc, scale=0.5), want_acc)


def test_what_has_no_split_form():
    x, w, out = _t(64, 68, seed=1), _t(64, 68, seed=2), torch.empty(64, 64, device="cuda")
    assert _split(x, w, out) != 0                                     # K not a multiple of 8
    x, w = _t(64, 72, seed=1), _t(64, 72, seed=2)
    assert _split(x.flatten()[1:1 + 63 * 72].view(63, 72), w, out[:63]) != 0  # off a 16-byte boundary
    assert _lib.lib().pg_gemm_fp32_scratch(8, 4096, 4096) == 0
    # and the products take such calls as before
    K, xs = 2052, _t(300, 2052, seed=3)
    ws = _t(2048, K, seed=4, scale=K ** -0.5)
    got = seq_ops.linear(xs, ws, torch.empty(300, 2048, device="cuda"))
    want = xs.double() @ ws.double().T
    assert ((got.double() - want).norm() / want.norm()).item() < 1e-6
