"""A routed feed-forward issued by one call against its launches one by one: the same kernels on the same rows, so the same bits; and the calls that keep the separate launches."""
import pytest
import torch

from paligemma_multimodal_system_b200 import mixers, seq_ops

pytestmark = pytest.mark.gpu


def _layer(D, experts, identity, top, F, shared, activation="relu2", **kw):
    ff = mixers.RoutedFeedForward(D, experts, identity, top, 1, 1, 2.5, F, shared, activation=activation, **kw)
    g = torch.Generator().manual_seed(3)
    ff.load(lambda name, shape: torch.randn(*shape, generator=g) * (shape[-1] ** -0.5 if len(shape) > 1 else 0.05), "")
    return ff


@pytest.mark.parametrize("T", [1, 63, 65, 200])
@pytest.mark.parametrize("kw", [dict(shared=512), dict(shared=0), dict(shared=520, shared_gate=True), dict(shared=0, activation="silu_glu"), dict(shared=0, activation="gelu", router_bias=True),
                                dict(shared=256, correction=False)])
@pytest.mark.parametrize("add", [False, True])
def test_same_bits_as_separate_launches(T, kw, add):
    prec = seq_ops.Precision(torch.bfloat16)
    ff = _layer(512, 6, 2, 3, 256, **kw)
    ff.pack(prec)
    g = torch.Generator(device="cuda").manual_seed(T)
    h = torch.randn(T, 520, generator=g, device="cuda").to(torch.bfloat16)[:, :512]  # (a view with a pitch)
    resid = torch.randn(T, 512, generator=g, device="cuda")
    assert ff._one_call(h, prec) is not None
    got = ff(h, None, prec, resid=resid.clone() if add else None)
    ff._one_call = lambda *a: None
    want = ff(h, None, prec, resid=resid.clone() if add else None)
    if kw["shared"] and T <= 128:  # the shared expert's products may add split parts in any order
        assert ((got - want).abs() <= 1e-5 * want.abs().max()).all()
    else:
        assert torch.equal(got, want)


def test_calls_that_keep_the_separate_launches():
    bf, f32 = seq_ops.Precision(torch.bfloat16), seq_ops.Precision(torch.float32)
    small, fits = _layer(128, 4, 0, 2, 64, 0), _layer(512, 6, 2, 3, 256, 512)
    glu = _layer(512, 6, 0, 2, 256, 256, activation="silu_glu")
    for ff in (small, fits, glu):
        ff.pack(bf)
    h = torch.randn(40, 512, device="cuda").to(torch.bfloat16)
    assert small._one_call(h[:, :128].contiguous(), bf) is None     # the smallest experts gather on the way
    assert glu._one_call(h, bf) is None                              # a gated shared expert
    assert fits._one_call(h.float(), f32) is None
    assert fits._one_call(h.flatten()[4:4 + 39 * 512].view(39, 512), bf) is None  # off a 16-byte boundary
    assert fits._one_call(torch.zeros(600, 512, device="cuda", dtype=torch.bfloat16), bf) is None  # dense runs
