"""Routed layers whose router outputs are all identity outputs: y = sum of the weights x h (+ the shared expert), no expert rows, no plan."""
import pytest
import torch

from paligemma_multimodal_system_b200 import mixers, seq_ops


def test_plan_without_experts_names_no_row(monkeypatch):
    """Every pair stays without an expert row, whatever the counts hold, and nothing is launched."""
    def refuse(*a):
        raise AssertionError("no plan kernel without experts")

    monkeypatch.setattr(seq_ops._lib, "lib", lambda: type("L", (), dict(pg_moe_plan=refuse, pg_moe_tile_rows=lambda: 64)))
    ids = torch.tensor([[0, 2], [1, 0], [2, 1]], dtype=torch.int32)
    plan = seq_ops.MoePlan(ids, torch.tensor([12345], dtype=torch.int32), 0)
    assert plan.pair_row.tolist() == [-1] * 6 and plan.pairs == 6 and plan.top == 2


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("shared", [0, 64])
@pytest.mark.parametrize("add", [False, True])
def test_identity_outputs_only(dtype, T, shared, add):
    D, n, top = 128, 4, 2
    ff = mixers.RoutedFeedForward(D, 0, n, top, 1, 1, 2.5, 256, shared)
    g = torch.Generator().manual_seed(3)
    w = {}

    def take(name, shape):
        w[name] = (torch.randn(*shape, generator=g) * (shape[-1] ** -0.5 if len(shape) > 1 else 0.05)).to(dtype).float()
        return w[name]

    ff.load(take, "")
    prec = seq_ops.Precision(dtype)
    ff.pack(prec)
    h = torch.randn(T, D, generator=g).to(dtype)
    resid = torch.randn(T, D, generator=g)
    got = ff(h.cuda(), None, prec, resid=resid.cuda() if add else None).cpu().double()
    hd = h.double()
    p = torch.softmax(hd @ w["router"].double().T, -1)
    chosen = torch.topk(p + w["correction"].double(), top, -1).indices
    pc = p.gather(1, chosen)
    want = (pc / pc.sum(-1, keepdim=True) * 2.5).sum(-1, keepdim=True) * hd  # (the weights of a token add up to the scale)
    if shared:
        mid = torch.relu(hd @ w["shared.up"].double().T) ** 2
        want = want + mid.to(dtype).double() @ w["shared.down"].double().T
    if add:
        want = want + resid.double()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 and shared else 1e-5  # (bf16: the shared expert's inner values are rounded once)
    assert ((got - want).abs() <= tol * (1 + want.abs())).all(), (got - want).abs().max()
