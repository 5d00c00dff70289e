"""fp32 matrix products (pg_gemm_simt, pg_gemm_simt_bias, pg_gemm_simt_batched with fp32 operands) against 64-bit products.

Bound per element: the k products are summed in at least two chains of at most ceil(K / 2) FMAs whose sums are added over at most 8 cluster ranks
and 32 lanes, so |error| <= (K / 2 + 48) 2^-24 sum_k |x w|; bias, scale and residual add three roundings of their own."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu


def _operands(T, F, K, seed, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K + pad, device="cuda", generator=g)[:, :K]
    w = torch.randn(F, K + pad, device="cuda", generator=g)[:, :K]
    return x, w


def _bound(x, w, K):
    return (K / 2 + 48) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("T", [1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128, 129, 300])
@pytest.mark.parametrize("F,K,pad", [(1, 1, 0), (33, 4, 0), (31, 127, 0), (64, 128, 4), (130, 1000, 3), (2048, 516, 0), (96, 8192, 0), (100, 2051, 0)])
def test_product(T, F, K, pad):
    x, w = _operands(T, F, K, T * 7 + F, pad)
    out = torch.full((T, F + 5), float("nan"), device="cuda")
    seq_ops.linear(x, w, out[:, :F])
    assert ((out[:, :F].double() - x.double() @ w.double().T).abs() <= _bound(x, w, K)).all()
    assert out[:, F:].isnan().all()


@pytest.mark.parametrize("T,F,K", [(3, 40, 1024), (16, 513, 4096), (40, 200, 2048), (200, 257, 300)])
def test_bias_scale_residual(T, F, K):
    x, w = _operands(T, F, K, 3)
    b, h = torch.randn(F, device="cuda"), torch.randn(T, F, device="cuda")
    want = h.double() + (x.double() @ w.double().T + b.double()) * 0.3
    bound = _bound(x, w, K) + 4 * 2.0 ** -24 * (want.abs() + h.double().abs() + b.double().abs())
    got = seq_ops.linear_add(x, w, h.clone(), bias=b, scale=0.3)
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("T,B,F,K", [(2, 32, 256, 64), (16, 3, 40, 2048), (70, 16, 64, 256), (19, 5, 33, 30)])
def test_batched(T, B, F, K):
    x, w = torch.randn(T, B, K + 8, device="cuda")[:, :, :K], torch.randn(B, F, K, device="cuda")
    out = torch.empty(T, B, F, device="cuda")
    seq_ops.linear_batched(x, w, out)
    want = torch.einsum("tbk,bfk->tbf", x.double(), w.double())
    bound = (K / 2 + 48) * 2.0 ** -24 * torch.einsum("tbk,bfk->tbf", x.double().abs(), w.double().abs())
    assert ((out.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("T", [4, 20, 150])
def test_same_result_twice(T):
    x, w = _operands(T, 2048, 4096, 11)
    a, b = (seq_ops.linear(x, w, torch.empty(T, 2048, device="cuda")) for _ in range(2))
    assert torch.equal(a, b)


def test_infinities_stay_in_their_rows():
    x, w = _operands(6, 70, 600, 5)
    x[2, 17] = float("inf")
    w[5, 3] = float("nan")
    out = seq_ops.linear(x, w, torch.empty(6, 70, device="cuda"))
    assert out[:, 5].isnan().all()
    keep = torch.ones(6, 70, dtype=torch.bool, device="cuda")
    keep[2], keep[:, 5] = False, False
    assert out[keep].isfinite().all() and not out[2].isfinite().any()


def test_no_rows_are_refused():
    w = torch.randn(8, 16, device="cuda")
    assert _lib.lib().pg_gemm_simt(w.data_ptr(), 16, w.data_ptr(), 16, w.data_ptr(), 8, 0, 8, 16, 1, 1, _lib.stream()) != 0


@pytest.mark.parametrize("T", [1, 4, 6, 7, 16])
@pytest.mark.parametrize("F,K", [(96, 64), (1000, 516), (2048, 8192), (4096, 2052)])
def test_weights_requested_ahead_of_the_rows(T, F, K):
    """In a step that says that weights follow, a few rows' product asks for its weights while the kernel in front writes the rows: the same sums bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(T + K)
    gu, w = torch.randn(T, 2 * K, generator=g, device="cuda"), torch.randn(F, K, generator=g, device="cuda")
    outs = []
    for on in (False, True):
        mid, out = torch.zeros(T, K, device="cuda"), torch.empty(T, F, device="cuda")
        if on:
            _lib.lib().pg_weights_follow(1)
        try:
            for _ in range(3):
                seq_ops.geglu(gu, mid)
                seq_ops.linear(mid, w, out)
        finally:
            if on:
                _lib.lib().pg_weights_follow(0)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    a = torch.nn.functional.gelu(gu[:, :K].double(), approximate="tanh") * gu[:, K:].double()
    # the sums' bound, and 2^-20 of every value for gelu's and the product's roundings
    want, mag = a @ w.double().T, a.abs() @ w.abs().double().T
    assert ((outs[1].double() - want).abs() <= ((K / 2 + 48) * 2.0 ** -24 + 2.0 ** -20) * mag).all()
