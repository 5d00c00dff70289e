"""Which kernels a ragged step takes, and what they are told of it (no device: the library is a stub that keeps its calls)."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops


class _Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append((name, a)) or 0


def _batch(ns):
    z = torch.zeros(len(ns), dtype=torch.int32)
    return seq_ops.StepBatch(T=sum(ns), E=len(ns), max_n=max(ns), min_n=min(ns), tokens=z, pos=z, row_entry=z, row0=z, n=z, ctx=z, slot=z, page_table=z.view(-1, 1), max_pages=1,
                             singles=sum(n == 1 for n in ns))


@pytest.fixture
def library(monkeypatch):
    library = _Library()
    monkeypatch.setattr(_lib, "lib", lambda: library)
    monkeypatch.setattr(_lib, "stream", lambda: 0)
    return library


BLOCKS, FMA, SCAN = "pg_linear_attn_blocks", "pg_linear_attn_chunked", "pg_linear_attn_scan"


@pytest.mark.parametrize("ns,H,dtype,want", [
    ([2000] + [1] * 40, 16, torch.bfloat16, [(FMA, 8, 1), (SCAN, 1, 0)]),
    ([2000] + [1] * 40, 24, torch.bfloat16, [(FMA, 8, 1), (SCAN, 1, 0)]),
    ([2000] + [1] * 40, 25, torch.bfloat16, [(BLOCKS, 8, 1), (SCAN, 1, 0)]),
    ([2000, 300], 32, torch.bfloat16, [(BLOCKS, 8, 2)]),
    ([2000], 32, torch.bfloat16, [(FMA, 8, 1)]),
    ([1] * 41, 32, torch.bfloat16, [(SCAN, 1, 0)]),
    ([2000] + [1] * 40, 16, torch.float32, [(FMA, 1, 0)]),
])
def test_linear_attention(library, monkeypatch, ns, H, dtype, want):
    """Single tokens own no blocks: the form and its sizes follow the entries that do."""
    b, d = _batch(ns), 64
    qkv, state, out = torch.zeros(b.T, 3 * H * d, dtype=dtype), torch.zeros(1, H, d, d), torch.zeros(b.T, H * d)
    monkeypatch.setattr(seq_ops, "_aligned", lambda t, n=16: True)
    seen = []

    def note(name):
        def call(*a):
            ops = _lib.LinearAttnOps.from_address(a[13])
            seen.append((name, ops.n_min, ops.portions))
            return 0
        return call

    for name in (BLOCKS, FMA, SCAN):
        setattr(library, name, note(name))
    seq_ops.linear_attn(qkv, state, torch.zeros(H), out, b, H, d, d)
    assert seen == want


@pytest.mark.parametrize("ns,portions", [([700] + [1] * 40, 1), ([700, 2], 2), ([1] * 5, 0)])
def test_short_convolution(library, ns, portions):
    b = _batch(ns)
    sec = seq_ops.ConvSections([dict(groups=1, size=8, xcol=0, ccol=0)])
    seq_ops.short_conv(torch.zeros(b.T, 8), torch.zeros(4, 8), torch.zeros(1, 3, 8), torch.zeros(b.T, 8), sec, b)
    (name, args), = library.calls
    assert name == "pg_short_conv_sized" and args[16:19] == (len(ns), max(ns), portions)


def test_a_step_is_described_in_the_order_that_it_was():
    """Fields that came later stand behind those that a caller may give by position."""
    import dataclasses
    names = [f.name for f in dataclasses.fields(seq_ops.StepBatch)]
    assert names == ["T", "E", "max_n", "tokens", "pos", "row_entry", "row0", "n", "ctx", "slot", "page_table", "max_pages", "singles", "max_single_ctx", "single_rows", "dense_row0", "dense_pages",
                     "dense_max_pages", "dense_rows", "dense_max_len", "shared", "min_n"]
