"""Token-major products at the edges of their tiles: 192-column tiles (CTA pair and one CTA), the choice between tile widths, feature tails and token remainders,
bf16 rows in whole 16-byte pieces and not.  Against 64-bit sums; bf16 operands, so a sum of K products of N(0, 1) x N(0, 1 / K) lies within 1e-4 before its rounding (2^-9)."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib

pytestmark = pytest.mark.gpu


def _t(*shape, seed, scale=1.0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _act(y, act):
    if act == 1:
        return torch.nn.functional.gelu(y, approximate="tanh")
    if act == 2:
        return torch.relu(y) ** 2
    return torch.nn.functional.gelu(y) if act == 6 else y


@pytest.fixture(autouse=True)
def _automatic_again():
    yield
    _lib.lib().pg_debug_set_gemm_bn(0)


# 2100 x 2560: pairs, 192 columns by rule; 1420 x 2048: one CTA, 192; 1420 x 1152: 128; 1500 x 640: 64; 4100 x 2560: pairs, 256; 1154 and 1160 features: tails of 2 and 8
@pytest.mark.parametrize("bn", [0, 192, 256])
@pytest.mark.parametrize("T,N,K", [(2100, 2560, 328), (1420, 2048, 264), (1420, 1152, 200), (1500, 640, 136), (4100, 2560, 192), (2049, 4304, 1152), (2305, 1160, 264), (1411, 1154, 264)])
def test_bf16_rows(bn, T, N, K):
    x, w, bias = _t(T, K, seed=1), _t(N, K, seed=2, scale=K ** -0.5), _t(N, seed=3, dtype=torch.float32)
    y = x.double() @ w.double().T + bias.double()
    _lib.lib().pg_debug_set_gemm_bn(bn)
    for act in (0, 1, 2, 6):
        whole = torch.full((T, N + 16), 7.0, device="cuda", dtype=torch.bfloat16)
        out = whole[:, 8:8 + N]
        _lib.gemm(x, w, out, mode=_lib.EPI_BF16, act_gelu=act, bias=bias, swap=0)
        want = _act(y, act)
        assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2e-3 * (1 if act == 1 else 0.2)).all()  # (tanh of the hardware: 2^-11 of the value's scale)
        assert (whole[:, :8] == 7).all() and (whole[:, 8 + N:] == 7).all()


@pytest.mark.parametrize("bn", [0, 192, 256])
@pytest.mark.parametrize("T,N,K", [(2100, 2560, 328), (1420, 2048, 264), (2305, 1160, 264), (8200, 1152, 136), (2561, 1154, 2056)])
def test_fp32_rows_with_residual(bn, T, N, K):
    x, w, bias, res = _t(T, K, seed=4), _t(N, K, seed=5, scale=K ** -0.5), _t(N, seed=6, dtype=torch.float32), _t(T, N, seed=7, dtype=torch.float32)
    want = x.double() @ w.double().T + bias.double() + res.double()
    _lib.lib().pg_debug_set_gemm_bn(bn)
    _lib.gemm(x, w, res, mode=_lib.EPI_F32, bias=bias, resid=res, swap=0)
    assert (res.double() - want).abs().max().item() < 1e-4
