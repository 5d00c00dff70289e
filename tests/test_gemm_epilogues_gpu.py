"""Every epilogue of the persistent tcgen05 kernels (gemm_tcgen05.cu) against 64-bit products: the one-CTA kernel with 64-, 128- and 256-wide tiles (the last with
four and with eight epilogue warps), the CTA-pair kernel (four and eight), the decode kernels of 16, 32, 64 and 128 tokens.

Bounds as in test_gemm_cluster_gpu.py: K 2^-23 sum_k |x w| for the sum, 2^-24 for every fp32 rounding, 2^-8 of a bf16 result, 2^-10 of the operands of a fast gelu / silu."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib

pytestmark = pytest.mark.gpu


def _operands(T, F, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(F, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    b = torch.randn(F, device="cuda", generator=g)
    xd, wd = x.double(), w.double()
    return x, w, b, xd @ wd.T, K * 2.0 ** -23 * (xd.abs() @ wd.abs().T)


def _check(got, want, bound):
    assert got.isfinite().all()
    assert ((got.double() - want).abs() <= bound).all()


ACTS = {0: lambda z: z, 1: lambda z: torch.nn.functional.gelu(z, approximate="tanh"), 2: lambda z: z.clamp(min=0) ** 2, 6: torch.nn.functional.gelu}
LIMIT, ALPHA = 1.5, 1.7


def _gated(kind, g, u):
    if kind == _lib.GLU_SILU:
        return g * torch.sigmoid(g) * u
    if kind == _lib.GLU_RELU:
        return g.clamp(min=0) * u
    if kind == _lib.GLU_CLAMPED:
        gc = g.clamp(max=LIMIT)
        return gc * torch.sigmoid(ALPHA * gc) * (u.clamp(-LIMIT, LIMIT) + 1)
    return torch.nn.functional.gelu(g, approximate="tanh") * u


def _run_gated(x, w, b, acc, bound, kind, swap):
    T, F = acc.shape
    z, e = (acc + (b.double() if b is not None else 0)).view(T, F // 128, 2, 64), bound.view(T, F // 128, 2, 64)
    g, u = z[:, :, 0], z[:, :, 1]
    want = _gated(kind, g, u)
    out = torch.full((T, F // 2), float("nan"), device="cuda", dtype=torch.bfloat16)
    _lib.gemm(x, w, out, mode=_lib.EPI_GEGLU, bias=b, act_gelu=kind, scale=LIMIT if kind == _lib.GLU_CLAMPED else 1.0, glu_alpha=ALPHA, swap=swap)
    err = 2 * (e[:, :, 0] * (u.abs() + 2) + e[:, :, 1] * (g.abs() + 2)) + 2.0 ** -8 * want.abs() + 2.0 ** -10 * (g * u).abs() + 2.0 ** -20 * (g.abs() + 1) * (u.abs() + 1)
    _check(out, want.reshape(T, -1), err.reshape(T, -1))


# (tokens, features, K): what pg_gemm_bf16 chooses for them above 1408 tokens
PROMPTS = [
    (1409, 512, 520),     # one CTA per tile, 64 wide (gated: 128)
    (1500, 1280, 520),    # 128 wide
    (1500, 2688, 520),    # 256 wide, eight epilogue warps
    (1500, 2688, 1544),   # 256 wide, four
    (1900, 2688, 520),    # CTA pairs, eight
    (1900, 2688, 2056),   # CTA pairs, four
]


@pytest.mark.parametrize("T,F,K", PROMPTS)
@pytest.mark.parametrize("act", sorted(ACTS))
def test_bf16_rows(T, F, K, act):
    F += 4  # a feature tail
    x, w, b, acc, bound = _operands(T, F, K, T + act)
    z = acc + b.double()
    out = torch.full((T, F + 4), float("nan"), device="cuda", dtype=torch.bfloat16)
    _lib.gemm(x, w, out[:, :F], mode=_lib.EPI_BF16, bias=b, act_gelu=act, swap=0)
    slope = 1.2 if act != 2 else 2 * z.abs() + 1
    want = ACTS[act](z)
    _check(out[:, :F], want, bound * slope + 2.0 ** -8 * want.abs() + (2.0 ** -10 * z.abs() if act == 1 else 0) + 1e-6)
    assert out[:, F:].isnan().all()


@pytest.mark.parametrize("T,F,K", PROMPTS)
def test_fp32_rows(T, F, K):
    x, w, b, acc, bound = _operands(T, F, K, T + 7)
    h = torch.randn(T, F, device="cuda")
    want = (acc + b.double()) * 0.5 + h.double()
    err = bound + 2.0 ** -22 * (want.abs() + h.double().abs() + b.double().abs())
    _check(_lib.gemm(x, w, torch.empty_like(h), mode=_lib.EPI_F32, bias=b, resid=h, scale=0.5, swap=0), want, err)
    for split in (1, 3):
        _check(_lib.gemm(x, w, h.clone(), mode=_lib.EPI_ATOMIC_F32, bias=b, scale=0.5, swap=0, split_k=split), want, err)


@pytest.mark.parametrize("T,F,K", PROMPTS)
@pytest.mark.parametrize("kind", [0, _lib.GLU_GELU, _lib.GLU_SILU, _lib.GLU_CLAMPED, _lib.GLU_RELU])
@pytest.mark.parametrize("bias", [False, True])
def test_gated_prompts(T, F, K, kind, bias):
    x, w, b, acc, bound = _operands(T, F, K, T * 3 + kind)
    _run_gated(x, w, b if bias else None, acc, bound, kind, 0)


@pytest.mark.parametrize("T", [1, 5, 16, 17, 32, 33, 40, 64, 65, 100, 128])
@pytest.mark.parametrize("kind", [0, _lib.GLU_GELU, _lib.GLU_SILU, _lib.GLU_CLAMPED, _lib.GLU_RELU])
@pytest.mark.parametrize("bias", [False, True])
def test_gated_decode(T, kind, bias):
    """256 tiles of 128 features: more than one wave of clusters, so the weight-streaming kernels take them."""
    x, w, b, acc, bound = _operands(T, 32768, 264, T * 5 + kind)
    _run_gated(x, w, b if bias else None, acc, bound, kind, 1)


@pytest.mark.parametrize("T", [5, 40, 130, 300, 1409])
def test_infinities_stay_in_their_rows(T):
    """Clustered, decode and one-CTA forms: an infinity in a token's row and a NaN in a feature's weights reach that row and that column alone, K and token tails included."""
    for F, K in ((516, 520), (32772, 72)):
        x, w, b, acc, bound = _operands(T, F, K, 9)
        x[3, 17], w[5, 3] = float("inf"), float("nan")
        keep = torch.ones(T, F, dtype=torch.bool, device="cuda")
        keep[3], keep[:, 5] = False, False
        for mode, dtype in ((_lib.EPI_F32, torch.float32), (_lib.EPI_BF16, torch.bfloat16)):
            out = _lib.gemm(x, w, torch.empty(T, F, device="cuda", dtype=dtype), mode=mode, swap=1 if T <= 128 else 0)
            assert out[:, 5].isnan().all() and not out[3].isfinite().any()
            assert ((out[keep].double() - acc[keep]).abs() <= (bound + 2.0 ** (-22 if dtype == torch.float32 else -8) * acc.abs())[keep]).all()
