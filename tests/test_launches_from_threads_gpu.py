"""Two host threads that run calls of one kernel with different amounts of shared memory: a launch must not depend on what the other thread asked for.  (ctypes drops the
interpreter lock, so the calls do interleave.)"""
import threading

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu


def _both(calls, rounds):
    """Runs every call `rounds` times on a thread and a stream of its own; the status codes that were not zero."""
    gate, bad = threading.Barrier(len(calls)), []

    def run(call):
        with torch.cuda.stream(torch.cuda.Stream()):
            st = _lib.stream()
            gate.wait()
            bad.extend(rc for rc in (call(st) for _ in range(rounds)) if rc != 0)

    threads = [threading.Thread(target=run, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return bad


def test_fp32_products():
    L, x = _lib.lib(), torch.randn(24, 512, device="cuda")
    ws = [torch.randn(f, 512, device="cuda") * 512 ** -0.5 for f in (1024, 32768)]  # one tile form, grids of less than one and of several CTAs per SM
    outs = [torch.zeros(24, w.shape[0], device="cuda") for w in ws]
    torch.cuda.synchronize()
    calls = [lambda st, w=w, o=o: L.pg_gemm_simt(x.data_ptr(), 512, w.data_ptr(), 512, o.data_ptr(), o.stride(0), 24, w.shape[0], 512, 1, 1, st) for w, o in zip(ws, outs)]
    assert _both(calls, 3000) == []
    for w, o in zip(ws, outs):
        want = x.double() @ w.double().T
        assert ((o.double() - want).norm() / want.norm()).item() < 1e-6


def test_single_token_attention():
    """Head groups whose query rows take 51 KB and 87 KB."""
    L, b = _lib.lib(), seq_ops.make_step_batch([dict(tokens=[1], ctx=40, slot=0, pages=[0])])
    calls, keep = [], []
    for H in (200, 340):
        q, k, v = (torch.randn(n, device="cuda").to(torch.bfloat16) for n in (H * 64, 64 * 64, 64 * 64))
        out = torch.zeros(1, H * 64, device="cuda", dtype=torch.bfloat16)
        keep.append((q, k, v, out))
        calls.append(lambda st, H=H, q=q, k=k, v=v, out=out: L.pg_attn_decode(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), 0, 0, out.data_ptr(), 0, b.row0.data_ptr(), b.n.data_ptr(), b.ctx.data_ptr(), b.page_table.data_ptr(), b.max_pages,
            64, b.E, 1, H, 1, 64, 64, 0.125, 0.0, 0, 0, 0, 0, 0, st))
    torch.cuda.synchronize()
    assert _both(calls, 2000) == []
    for q, k, v, out in keep:
        kk, vv = k.view(64, 64)[:41].double(), v.view(64, 64)[:41].double()
        want = torch.softmax(q.view(-1, 64).double() @ kk.T * 0.125, -1) @ vv
        assert ((out.view(-1, 64).double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
