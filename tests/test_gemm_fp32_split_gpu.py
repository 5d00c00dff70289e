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
