"""Calls whose kernels bound their waits may be captured before anything has run on the device."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import torch
from vllm_b200.ops import cuda as cu, ref
from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout
g = torch.Generator(device="cuda").manual_seed(0)
x = torch.randn(1400, 256, device="cuda", generator=g).bfloat16()
wq, ws = ref.block_quant_weight_fp8(torch.randn(4096, 256, device="cuda", generator=g), 128)
ws = ws.contiguous()
xq, xs = cu.per_token_group_quant_fp8(x, 128, col_major=True)
w = torch.randn(2, 64, 256, device="cuda", generator=g).bfloat16()
offs = torch.tensor([0, 700, 1400], dtype=torch.int32, device="cuda")
q, cache, md = _mk_attn_case(2, 8, 2, 128, 64, [70, 40], [70, 40])
md.kv_vt, cache = True, _to_tc_layout(cache)
assert cu.fp8_rows(1400, 4096, 256) and not cu._kernel_error
run = lambda: (cu.gemm_fp8_block(xq, xs, wq, ws), cu.gemm_grouped(x, w, offs), cu.paged_attention(q, cache, md, 0.1))
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    got = run()
graph.replay()
torch.cuda.synchronize()
assert all(torch.equal(a, b) for a, b in zip(got, run()))
"""


def test_first_call_in_a_capture():
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
