"""Slots of the cache that are not a sequence's (behind its end, in front of its window, pages of others) may hold anything."""
import math

import pytest
import torch

from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout, cu
from vllm_b200.ops import ref

pytestmark = pytest.mark.gpu


def _poison(cache, bt, seq_lens, firsts):
    """NaN and infinities in all slots but positions ``firsts`` .. ``seq_lens`` - 1 of each sequence; cache [blocks, ..., slots, width] by slot."""
    bs = cache.shape[-2]
    keep = torch.zeros(cache.shape[0], bs, dtype=torch.bool, device=cache.device)
    for row, n, a in zip(bt.tolist(), seq_lens, firsts):
        for pos in range(max(a, 0), n):
            keep[row[pos // bs], pos % bs] = True
    bad = torch.tensor([float("inf"), float("nan"), float("-inf")], device=cache.device, dtype=cache.dtype)
    flat = torch.arange(keep.numel(), device=cache.device).view(keep.shape) % 3
    mask = keep.view(keep.shape[0], *[1] * (cache.dim() - 3), bs, 1)
    return torch.where(mask, cache, bad[flat].view(*mask.shape))


def _close(got, want):
    # a rounding of the result, and of the weights where they keep 16 bits: test_prompt_attention_gpu.py
    assert bool(got.isfinite().all())
    assert float((got.double() - want.double()).norm() / want.double().norm()) < 2 ** -8


@pytest.mark.parametrize("lens", [([17, 64, 300, 130, 1, 513, 129], [17, 64, 172, 1, 1, 513, 2]), ([1031, 700, 64, 2500, 257], [1031, 573, 1, 1400, 129])],
                         ids=["one", "two"])                                     # query tiles per CTA
@pytest.mark.parametrize("Hq,Hkv,window", [(32, 8, None), (32, 8, 100), (4, 4, 700), (8, 1, 129)])
@pytest.mark.parametrize("cap", [0.0, 50.0])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prompts(lens, Hq, Hkv, window, cap, dtype):
    seq_lens, q_lens = lens
    q, cache, md = _mk_attn_case(len(seq_lens), Hq, Hkv, 128, 64, seq_lens, q_lens, dtype=dtype, seed=4)
    md.kv_vt = True
    want = ref.paged_attention(q, cache, md.block_table, md.seq_lens_cpu, md.query_start_loc_cpu, 0.1, sliding_window=window, logits_soft_cap=cap)
    bad = _poison(cache, md.block_table, seq_lens, [n - m + 1 - window if window else 0 for n, m in zip(seq_lens, q_lens)])
    _close(cu().paged_attention(q, _to_tc_layout(bad), md, 0.1, window, cap), want)


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (8, 1), (4, 4), (32, 1)])
@pytest.mark.parametrize("window", [None, 100])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("cap", [0.0, 50.0])
def test_decode(Hq, Hkv, window, splits, cap):
    seq_lens = [1, 63, 64, 65, 127, 128, 129, 1000, 257, 5]
    q, cache, md = _mk_attn_case(len(seq_lens), Hq, Hkv, 128, 64, seq_lens, [1] * len(seq_lens))
    md.num_splits, md.kv_vt = splits, True
    want = ref.paged_attention(q, cache, md.block_table, md.seq_lens_cpu, md.query_start_loc_cpu, 0.2, sliding_window=window, logits_soft_cap=cap)
    bad = _poison(cache, md.block_table, seq_lens, [n - window if window else 0 for n in seq_lens])
    _close(cu().paged_attention(q, _to_tc_layout(bad), md, 0.2, window, cap), want)


@pytest.mark.parametrize("H,R,P,page", [(16, 512, 64, 64), (40, 512, 64, 32), (5, 136, 16, 16), (16, 256, 0, 128)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("splits", [1, 3])
def test_latents(H, R, P, page, window, wide, splits):
    lens = [1, 63, 64, 65, 200, 1030]
    g = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    n = -(-max(lens) // page)
    cache, q, qp = rnd(len(lens) * n + 3, page, R + P), rnd(len(lens), H, R), rnd(len(lens), H, P) if P else None
    bt = torch.randperm(len(lens) * n, device="cuda", generator=g).int().view(len(lens), n)
    want = []
    for i, m in enumerate(lens):
        kv = cache[bt[i].long()].view(-1, R + P)[max(m - window, 0) if window else 0:m].double()
        w = ((q[i] if qp is None else torch.cat([q[i], qp[i]], -1)).double() @ kv.t() / math.sqrt(R)).softmax(-1)
        want.append(w @ kv[:, :R])
    bad = _poison(cache, bt, lens, [m - window if window else 0 for m in lens])
    got = cu().mla_decode_tc(q, qp, bad, bt, torch.tensor(lens, dtype=torch.int32, device="cuda"), 1 / math.sqrt(R), max(lens), splits,
                             sliding_window=window or None, wide=wide)
    _close(got, torch.stack(want))
