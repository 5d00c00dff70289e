"""Calls on a machine without a GPU end with an error that the caller can catch."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _child(code):
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True, timeout=300)


def test_plans_need_no_device():
    r = _child("""
from paligemma_multimodal_system_b200 import _lib
L = _lib.lib()
for T, F, K in ((300, 512, 2048), (100000, 64, 64), (40, 32000, 2048)):
    assert L.pg_gemm_fp32_scratch(T, F, K) >= 0
""")
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("call", [
    "L.pg_gemm_fp32_split(a, 2048, a, 2048, a, 512, 0, 0, 1.0, 300, 512, 2048, a, 1 << 30, 0)",
    "L.pg_gemm_simt(a, 512, a, 512, a, 64, 40, 64, 512, 1, 1, 0)",
    "L.pg_gemm_bf16(a, 512, a, 512, a, 2048, 0, 0, 0, 1500, 2048, 512, 0, 1, 1.0, 0, 1, 0)",
    "L.pg_gemm_bf16(a, 2048, a, 2048, a, 2048, 0, 0, 0, 1000, 2048, 2048, 0, 1, 1.0, 0, 1, 0)",
    "L.pg_gemm_bf16(a, 512, a, 512, a, 2048, 0, 0, 0, 9000, 2048, 512, 1, 0, 1.0, 0, 1, 0)",
])
def test_products_return_an_error(call):
    r = _child(f"""
from paligemma_multimodal_system_b200 import _lib
L, a = _lib.lib(), 1 << 20  # (an address that nothing reads: no launch gets that far)
assert {call} != 0
""")
    assert r.returncode == 0, r.stderr[-2000:]


def test_fp32_linear_raises_on_host_tensors():
    r = _child("""
import torch
from paligemma_multimodal_system_b200 import seq_ops
try:
    seq_ops.linear(torch.randn(300, 2048), torch.randn(512, 2048), torch.empty(300, 512))
except RuntimeError:
    raise SystemExit(0)
raise SystemExit("no error")
""")
    assert r.returncode == 0, r.stderr[-2000:]
