"""Prompt and decode attention on the tensor cores: one and two query tiles per CTA, capped scores, edges of tiles, windows."""
import math

import pytest
import torch

from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout, cu
from vllm_b200.ops import ref

pytestmark = pytest.mark.gpu

# 16-bit results are off by at most 2^-9 of each value (bf16; fp16 2^-12), 16-bit weights by as much of each product: in the 2-norm the two add
# up to less than 2^-8.  Capped scores keep the weights in 32 bits: the rounding of the result is all that is left, below 2^-9.
LIMIT = {False: 2 ** -8, True: 2 ** -9}

SHORT = ([17, 64, 300, 130, 1, 513, 129], [17, 64, 172, 1, 1, 513, 2])          # fewer tiles than SMs: one per CTA
LONG = ([1031, 700, 64, 2500, 257], [1031, 573, 1, 1400, 129])                   # more: two, some CTAs with one


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("lens", [SHORT, LONG], ids=["one", "two"])
@pytest.mark.parametrize("Hq,Hkv,window", [(32, 8, None), (32, 8, 100), (4, 4, 700), (8, 1, None), (16, 8, 129)])
@pytest.mark.parametrize("cap", [0.0, 50.0, 2.0])
def test_prompts(lens, Hq, Hkv, window, cap):
    seq_lens, q_lens = lens
    q, cache, md = _mk_attn_case(len(seq_lens), Hq, Hkv, 128, 64, seq_lens, q_lens, seed=11)
    md.kv_vt = True
    scale = 2.0 / math.sqrt(128)                                                 # cap 2: most scores are beyond it
    got, lse = cu().paged_attention(q, _to_tc_layout(cache), md, scale, window, cap, return_lse=True)
    want, lse_w = ref.paged_attention(q, cache, md.block_table, md.seq_lens_cpu, md.query_start_loc_cpu, scale, sliding_window=window,
                                      logits_soft_cap=cap, return_lse=True)
    assert _rel(got, want) < LIMIT[cap > 0], _rel(got, want)
    assert _rel(lse, lse_w) < 1e-5
    cu().check_kernel_error(q.device)


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (8, 1), (4, 4), (16, 1), (32, 1)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cap", [50.0, 2.0])
def test_capped_decode(Hq, Hkv, splits, dtype, cap):
    seq_lens = [1, 63, 64, 65, 127, 128, 129, 1000, 257, 5]
    q, cache, md = _mk_attn_case(len(seq_lens), Hq, Hkv, 128, 64, seq_lens, [1] * len(seq_lens), dtype=dtype)
    md.num_splits, md.kv_vt = splits, True
    got = cu().paged_attention(q, _to_tc_layout(cache), md, 0.2, 300, cap)
    want = ref.paged_attention(q, cache, md.block_table, md.seq_lens_cpu, md.query_start_loc_cpu, 0.2, sliding_window=300, logits_soft_cap=cap)
    assert _rel(got, want) < LIMIT[True], _rel(got, want)
    cu().check_kernel_error(q.device)
