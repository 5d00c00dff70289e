"""The norms that keep a row in one warp's registers: every row width they are built for, an odd number of rows, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", range(128, 2049, 128))
def test_widths(D):
    from paligemma_multimodal_system_b200 import _lib
    rows, eps = 1027, 1e-6
    g = torch.Generator(device="cuda").manual_seed(D)
    x = torch.randn(rows, D, generator=g, device="cuda") * 3 + 0.5
    w, b = (torch.randn(D, generator=g, device="cuda") for _ in range(2))
    y, f = torch.empty(rows, D, device="cuda", dtype=torch.bfloat16), torch.empty(rows, D, device="cuda")
    xd = x.double()
    m = xd.mean(-1, keepdim=True)
    want = (xd - m) / torch.sqrt(((xd - m) ** 2).mean(-1, keepdim=True) + eps) * w.double() + b.double()
    _lib.layernorm(x, w, b, eps, out_bf16=y)
    _lib.layernorm(x, w, b, eps, out_f32=f)
    # sums of up to 2048 fp32 values: 2^-20 of the normalised values (up to 5 here) before the weight; bf16 rounds by 2^-9
    assert ((f.double() - want).abs() <= 2.0 ** -19 * (1 + want.abs()) * 5).all()
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all()
    _lib.rmsnorm(x, w, y, eps)
    want = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + eps) * (1 + w.double())
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all()


@pytest.mark.parametrize("rows", [1, 300])
@pytest.mark.parametrize("D", [4, 100, 128, 1152, 2044, 2048, 2052, 4096, 5000, 8192])
@pytest.mark.parametrize("shift", [0, 1])
def test_few_rows(rows, D, shift):
    """A row in a block's registers, and weights off 16 bytes: in shared memory."""
    from paligemma_multimodal_system_b200 import _lib
    eps = 1e-6
    g = torch.Generator(device="cuda").manual_seed(D)
    x = torch.randn(rows, D, generator=g, device="cuda") * 3 + 0.5
    w, b = (torch.randn(D + 1, generator=g, device="cuda")[shift:][:D] for _ in range(2))
    y, f = torch.empty(rows, D, device="cuda", dtype=torch.bfloat16), torch.empty(rows, D, device="cuda")
    xd = x.double()
    m = xd.mean(-1, keepdim=True)
    want = (xd - m) / torch.sqrt(((xd - m) ** 2).mean(-1, keepdim=True) + eps) * w.double() + b.double()
    _lib.check(_lib.lib().pg_layernorm(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), f.data_ptr(), rows, D, eps, _lib.stream()), "pg_layernorm")
    # as above; a row of four values may lie near its mean: its variance carries the error of the mean, 2^-22 of the row's values
    tol = 2.0 ** -19 * 5 if D > 4 else 2.0 ** -12
    assert ((f.double() - want).abs() <= tol * (1 + want.abs())).all()
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + tol).all()
    _lib.check(_lib.lib().pg_rmsnorm(x.data_ptr(), w.data_ptr(), y.data_ptr(), rows, D, eps, _lib.stream()), "pg_rmsnorm")
    want = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + eps) * (1 + w.double())
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all()


@pytest.mark.parametrize("rows", [1, 300])
@pytest.mark.parametrize("D", [4, 100, 1020, 1024, 1028, 1152, 2048, 2052, 4096, 4100, 8192])
def test_bits_do_not_depend_on_where_weights_lie(rows, D):
    """The form with the row in registers sums in the order of the one in shared memory, which weights off 16 bytes take."""
    from paligemma_multimodal_system_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(D + rows)
    x = torch.randn(rows, D, generator=g, device="cuda") * 3 + 0.5
    w, b = (torch.randn(D, generator=g, device="cuda") for _ in range(2))
    res = []
    for shift in (0, 1):
        ws, bs = (torch.cat([t.new_zeros(shift), t])[shift:] for t in (w, b))
        f, y, z = torch.empty(rows, D, device="cuda"), *(torch.empty(rows, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        _lib.check(_lib.lib().pg_layernorm(x.data_ptr(), ws.data_ptr(), bs.data_ptr(), y.data_ptr(), f.data_ptr(), rows, D, 1e-6, _lib.stream()), "pg_layernorm")
        _lib.check(_lib.lib().pg_rmsnorm(x.data_ptr(), ws.data_ptr(), z.data_ptr(), rows, D, 1e-6, _lib.stream()), "pg_rmsnorm")
        res.append((f, y, z))
    for a, c in zip(*res):
        assert torch.equal(a, c)
