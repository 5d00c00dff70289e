"""bf16 products refuse host tensors before a launch: their addresses would go into a tensor map as device addresses."""
import types

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops


@pytest.fixture(autouse=True)
def no_launch(monkeypatch):
    monkeypatch.setattr(_lib, "lib", lambda: pytest.fail("a launch was reached"))
    monkeypatch.setattr(_lib, "stream", lambda: 0)


@pytest.mark.parametrize("T", [1, 128, 129])
@pytest.mark.parametrize("out,bias", [(torch.float32, False), (torch.float32, True), (torch.bfloat16, False)])
def test_linear(T, out, bias):
    x, w = torch.zeros(T, 64, dtype=torch.bfloat16), torch.zeros(16, 64, dtype=torch.bfloat16)
    with pytest.raises(AssertionError):
        seq_ops.linear(x, w, torch.zeros(T, 16, dtype=out), bias=torch.zeros(16) if bias else None)


def test_residual():
    with pytest.raises(AssertionError):
        _lib.gemm_residual(torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(16, 64, dtype=torch.bfloat16), torch.zeros(4, 16))


def test_routed_products():
    D, F, n, pairs = 64, 32, 2, 6
    plan = types.SimpleNamespace(pairs=pairs, top=2, max_tiles=3, sorted_pair=torch.zeros(pairs, dtype=torch.int32), offsets=torch.zeros(n + 1, dtype=torch.int32),
                                 plan=torch.zeros(13, dtype=torch.int32))
    b = dict(dtype=torch.bfloat16)
    with pytest.raises(AssertionError):
        seq_ops.moe_products(torch.zeros(3, D, **b), plan, torch.zeros(n, F, D, **b), torch.zeros(n, D, F, **b), torch.zeros(pairs, D, **b), torch.zeros(pairs, F, **b),
                             torch.zeros(pairs, D), seq_ops.ACT_RELU2)
