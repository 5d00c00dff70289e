"""Products of a moderate number of tokens (gemm_cluster.cu, chosen by pg_gemm_bf16 for token-major calls) against 64-bit products.

Bound per element: bf16 products are exact in fp32, the tensor core adds them with at most one unit in the last place per addition, so the sum is
within K 2^-23 sum_k |x w|; an fp32 result adds four roundings, a bf16 result 2^-8 of itself, gelu / silu in their fast forms 2^-10 of the operands."""
import json

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

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


# token counts around the 16-, 32-, 128-, 256- and 384-token edges; feature and K tails; one to eight CTAs that share K
@pytest.mark.parametrize("T", [1, 15, 16, 129, 255, 256, 257, 263, 384, 385, 770, 1408])
@pytest.mark.parametrize("F,K", [(4, 8), (100, 64), (1152, 1152), (132, 72), (2048, 4304), (640, 520)])
def test_fp32_bias_residual(T, F, K):
    x, w, b, acc, bound = _operands(T, F, K, T + F)
    h = torch.randn(T, F, device="cuda")
    want = (acc + b.double()) * 0.5 + h.double()
    out = _lib.gemm(x, w, h.clone(), mode=_lib.EPI_F32, bias=b, resid=h, scale=0.5, swap=0)
    _check(out, want, bound + 2.0 ** -22 * (want.abs() + h.double().abs() + b.double().abs()))
    more = _lib.gemm(x, w, h.clone(), mode=_lib.EPI_ATOMIC_F32, bias=b, scale=0.5, swap=0, split_k=3)
    _check(more, want, bound + 2.0 ** -22 * (want.abs() + h.double().abs() + b.double().abs()))
    assert torch.equal(out, _lib.gemm(x, w, h.clone(), mode=_lib.EPI_F32, bias=b, resid=h, scale=0.5, swap=0))


@pytest.mark.parametrize("T", [130, 257, 300, 900])
@pytest.mark.parametrize("act,f", [(0, lambda z: z), (1, lambda z: torch.nn.functional.gelu(z, approximate="tanh")), (2, lambda z: z.clamp(min=0) ** 2), (6, torch.nn.functional.gelu)])
def test_bf16_activations(T, act, f):
    x, w, b, acc, bound = _operands(T, 516, 696, T + act)
    z = acc + b.double()
    out = torch.full((T, 520), float("nan"), device="cuda", dtype=torch.bfloat16)
    _lib.gemm(x, w, out[:, :516], mode=_lib.EPI_BF16, bias=b, act_gelu=act, swap=0)
    slope = 1.2 if act != 2 else 2 * z.abs() + 1
    _check(out[:, :516], f(z), bound * slope + 2.0 ** -8 * f(z).abs() + (2.0 ** -10 * z.abs() if act == 1 else 0) + 1e-6)
    assert out[:, 516:].isnan().all()


@pytest.mark.parametrize("T", [16, 200, 263, 1024])
@pytest.mark.parametrize("kind", [_lib.GLU_GELU, _lib.GLU_SILU, _lib.GLU_CLAMPED, _lib.GLU_RELU])
def test_gated_units(T, kind):
    F, K = 384, 1032
    x, w, b, acc, bound = _operands(T, F, K, T * 3 + kind)
    z, e = (acc + b.double()).view(T, F // 128, 2, 64), bound.view(T, F // 128, 2, 64)
    g, u = z[:, :, 0], z[:, :, 1]
    limit, alpha = 1.5, 1.7
    if kind == _lib.GLU_GELU:
        want = torch.nn.functional.gelu(g, approximate="tanh") * u
    elif kind == _lib.GLU_SILU:
        want = g * torch.sigmoid(g) * u
    elif kind == _lib.GLU_RELU:
        want = g.clamp(min=0) * u
    else:
        gc, uc = g.clamp(max=limit), u.clamp(-limit, limit)
        want = gc * torch.sigmoid(alpha * gc) * (uc + 1)
    out = torch.empty(T, F // 2, device="cuda", dtype=torch.bfloat16)
    _lib.gemm(x, w, out, mode=_lib.EPI_GEGLU, bias=b, act_gelu=kind, scale=limit if kind == _lib.GLU_CLAMPED else 1.0, glu_alpha=alpha, swap=0)
    bound = 2 * (e[:, :, 0] * (u.abs() + 2) + e[:, :, 1] * (g.abs() + 2)) + 2.0 ** -8 * want.abs() + 2.0 ** -10 * (g * u).abs() + 2.0 ** -20 * (g.abs() + 1) * (u.abs() + 1)
    _check(out, want.reshape(T, -1), bound.reshape(T, -1))


@pytest.mark.parametrize("T", [140, 512])
def test_row_map_and_table(T):
    F, K, N = 256, 640, 70
    x, w, b, acc, bound = _operands(T, F, K, T)
    rows = torch.randperm(T + 9, device="cuda")[:T].to(torch.int32)
    out = torch.full((T + 9, F), float("nan"), device="cuda")
    _lib.gemm(x, w, out, mode=_lib.EPI_F32, bias=b, scale=0.25, swap=0, out_row_map=rows)
    want = (acc + b.double()) * 0.25
    _check(out[rows.long()], want, bound + 2.0 ** -22 * (want.abs() + b.double().abs()))
    assert int(out.isnan().all(1).sum()) == 9
    table = torch.randn(N, F, device="cuda")
    out = torch.empty(T, F, device="cuda")
    _lib.gemm(x, w, out, mode=_lib.EPI_F32, bias=b, resid=table, resid_row_mod=N, swap=0)
    want = acc + b.double() + table.double()[torch.arange(T, device="cuda") % N]
    _check(out, want, bound + 2.0 ** -21 * (want.abs() + 4))


@pytest.mark.parametrize("T,F,K", [(16, 256, 512), (40, 640, 2048), (300, 512, 1024), (129, 1152, 4304)])
def test_clustered_ctas_have_an_sm_to_themselves(T, F, K, tmp_path):
    """A CTA that shares K with others holds tensor memory while it waits for them, so no second one may fit beside it: its launch asks for more than half of
    an SM's 228 KB of shared memory (1 KB a CTA belongs to the system)."""
    x, w, b, acc, bound = _operands(T, F, K, 1)
    out = torch.empty(T, F, device="cuda")
    _lib.gemm(x, w, out, mode=_lib.EPI_F32, swap=0)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        _lib.gemm(x, w, out, mode=_lib.EPI_F32, swap=0)
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    launches = [e["args"] for e in json.load(open(tmp_path / "trace.json"))["traceEvents"] if "gemm_cluster_kernel<true" in e.get("name", "")]
    assert launches and all(2 * (a["shared memory"] + 1024) > 228 * 1024 for a in launches)
    _check(out, acc, bound + 2.0 ** -22 * acc.abs())


@pytest.mark.parametrize("T", [5, 100, 263, 700])
def test_residual_buffers_may_be_larger(T):
    """gemm_residual adds to the first rows and columns of the stream it is given."""
    x, w, b, acc, bound = _operands(T, 256, 640, T)
    h = torch.randn(T + 3, 260, device="cuda")
    was = h.clone()
    _lib.gemm_residual(x, w, h, bias=b, scale=0.5)
    want = was[:T, :256].double() + (acc + b.double()) * 0.5
    _check(h[:T, :256], want, bound + 2.0 ** -21 * (want.abs() + was[:T, :256].double().abs() + b.double().abs()))
    assert torch.equal(h[T:], was[T:]) and torch.equal(h[:, 256:], was[:, 256:])
    with pytest.raises(AssertionError):
        _lib.gemm_residual(x, w, h[:T - 1], bias=b)


@pytest.mark.parametrize("F,K", [(64, 4104), (256, 8192), (512, 1024), (12288, 1640)])
def test_one_row_of_any_pitch(F, K):
    """The one row of a one-token product may come with any row pitch (a view of a column, an expanded row), also where its sums are split."""
    x, w, b, acc, bound = _operands(1, F, K, F)
    for pitch in (0, 8, F, 2 * F):
        out = torch.full((2 * F,), float("nan"), device="cuda")
        seq_ops.linear(x, w, out.as_strided((1, F), (pitch, 1)))
        _check(out[:F].view(1, F), acc, bound + 2.0 ** -22 * acc.abs())
        assert out[F:].isnan().all()


@pytest.mark.parametrize("T,F,K,split", [(200, 256, 512, 1), (300, 512, 1024, 4), (1400, 260, 640, 3)])
def test_atomic_accumulation_from_several_streams(T, F, K, split):
    """PG_EPI_ATOMIC_F32 outputs may be shared: sums of small whole numbers are exact in any order, so none may be lost."""
    xs, ws = (torch.randint(-2, 3, (8, n, K), device="cuda").bfloat16() for n in (T, F))
    out = torch.zeros(T, F, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    for i in range(8):
        with torch.cuda.stream(streams[i % 4]):
            _lib.gemm(xs[i], ws[i], out, mode=_lib.EPI_ATOMIC_F32, swap=0, split_k=split)
    torch.cuda.synchronize()
    assert torch.equal(out.double(), torch.einsum("itk,ifk->tf", xs.double(), ws.double()))


def _kernels(call):
    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return " ".join(e.key for e in prof.key_averages())


def test_tuning_switches_reach_the_persistent_kernels():
    L = _lib.lib()
    x, w, b, acc, bound = _operands(300, 512, 640, 2)
    out = torch.empty(300, 512, device="cuda", dtype=torch.bfloat16)
    few = torch.empty(5, 512, device="cuda", dtype=torch.bfloat16)
    prompt = lambda: _lib.gemm(x, w, out, mode=_lib.EPI_BF16, swap=0)
    assert "gemm_cluster_kernel" in _kernels(prompt)
    try:
        for bn in (64, 128, 256):
            assert L.pg_debug_set_gemm_bn(bn) == 0 and f"gemm_tcgen05_kernel<{bn}" in _kernels(prompt)
            _check(out, acc, bound + 2.0 ** -8 * acc.abs())
        L.pg_debug_set_gemm_bn(0)
        L.pg_debug_set_gemm_pair(0, 0)  # one CTA per tile only
        assert "gemm_tcgen05_kernel" in _kernels(prompt)
        L.pg_debug_set_gemm_pair(1, 1)  # pairs from one tile on
        assert L.pg_debug_set_gemm_bn(256) == 0 and "gemm_pair_kernel" in _kernels(prompt)
        _check(out, acc, bound + 2.0 ** -8 * acc.abs())
        L.pg_debug_set_gemm_bn(0)
        L.pg_debug_set_gemm_pair(1, 74)
        stamps = torch.zeros(64 * 8, device="cuda", dtype=torch.int64)
        L.pg_debug_set_gemm_trace(stamps.data_ptr())
        prompt()
        _lib.gemm(x[:5], w, few, mode=_lib.EPI_BF16, swap=1)
        torch.cuda.synchronize()
        assert (stamps.view(64, 8)[:2, 0] > 0).all()
    finally:
        L.pg_debug_set_gemm_bn(0)
        L.pg_debug_set_gemm_pair(1, 74)
        L.pg_debug_set_gemm_trace(0)
    assert "gemm_cluster_kernel" in _kernels(prompt)
