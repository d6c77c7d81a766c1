"""Prompt and decode attention on the tensor cores: one and two query tiles per CTA, capped scores, edges of tiles, windows."""
import math

import pytest
import torch

from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout, cu

pytestmark = pytest.mark.gpu

# Rounding to bf16 (8 bits of significand) is off by at most 2^-8 of a value, to fp16 by 2^-11; an error spread evenly over a unit in the last
# place has an RMS of 1 / sqrt(12) of it, which over values as frequent at every scale (mean square of the significand 2.16) is 2^-9.35 or 2^-12.35
# of them in the 2-norm.  Capped scores (and split, wide weights) keep 16 more bits of the weights, so that is all there is; 16-bit weights
# are off by as much again, independently: 2^-8.85 and 2^-11.85.  The limits lie between and above these.
LIMIT = {(False, torch.bfloat16): 2 ** -8, (True, torch.bfloat16): 2 ** -9, (False, torch.float16): 2 ** -11, (True, torch.float16): 2 ** -12}


def _exact(q, cache, md, scale, window, cap):
    """Attention over the pages in 64 bits: results and natural logarithms of the weights' sums."""
    outs, lses = [], []
    qsl, lens = md.query_start_loc_cpu.tolist(), md.seq_lens_cpu.tolist()
    for b, n in enumerate(lens):
        qi = q[qsl[b]:qsl[b + 1]].double()
        rows = cache[md.block_table[b].long()].transpose(0, 1).transpose(2, 3).flatten(1, 2)[:, :n].double()      # [2, n, heads, D]
        k, v = (x.repeat_interleave(qi.shape[1] // x.shape[1], 1) for x in rows)
        s = torch.einsum("qhd,khd->hqk", qi, k) * scale
        if cap:
            s = torch.tanh(s / cap) * cap
        pos, key = torch.arange(n - len(qi), n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
        s = s.masked_fill((key > pos) | (key <= pos - (window or n + 1)), float("-inf"))
        outs.append(torch.einsum("hqk,khd->qhd", s.softmax(-1), v))
        lses.append(torch.logsumexp(s, -1).t())
    return torch.cat(outs), torch.cat(lses)


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
    want, lse_w = _exact(q, cache, md, scale, window, cap)
    assert _rel(got, want) < LIMIT[cap > 0, q.dtype], _rel(got, want)
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
    want, _ = _exact(q, cache, md, 0.2, 300, cap)
    assert _rel(got, want) < LIMIT[True, dtype], _rel(got, want)
    cu().check_kernel_error(q.device)


@pytest.mark.parametrize("heads", [3, 32], ids=["one", "two"])                  # tiles per CTA
@pytest.mark.parametrize("dim,rot,vdim", [(128, 64, 128), (64, 0, 64), (24, 8, 40), (128, 0, 72)])
@pytest.mark.parametrize("split", [False, True])
def test_expanded_keys(heads, dim, rot, vdim, split):
    """Keys and values as columns of one matrix, key rows of a request behind a gap of zeros."""
    q_lens, seq_lens = [1, 127, 128, 129, 300, 513, 17], [200, 127, 640, 129, 301, 513, 17]
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    T = sum(q_lens)
    start = [0]
    for n in seq_lens:
        start.append(start[-1] + -(-n // 128) * 128)
    q, kv, kr = rnd(T, heads, dim + rot), rnd(start[-1], heads, dim + vdim), rnd(start[-1], max(rot, 8))
    for s, n, e in zip(start, seq_lens, start[1:]):
        kv[s + n:e], kr[s + n:e] = 0, 0
    out = torch.full((T, heads, vdim), float("nan"), device="cuda", dtype=torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    cu_q = [sum(q_lens[:i]) for i in range(len(q_lens) + 1)]
    cu().mla_prefill(q, kv[..., :dim], kv[..., dim:], out, i32(cu_q[:-1]), i32(q_lens), i32(seq_lens), i32(start), 0, max(q_lens), 0.1,
                     kr[:, :rot] if rot else None, split=split)
    cu().check_kernel_error(q.device)
    want = []
    for a, ql, s, n in zip(cu_q, q_lens, start, seq_lens):
        k = torch.cat([kv[s:s + n, :, :dim], kr[s:s + n, None, :rot].expand(-1, heads, -1)], -1).double()
        x = torch.einsum("qhd,khd->hqk", q[a:a + ql].double(), k) * 0.1
        x = x.masked_fill(torch.arange(n, device="cuda")[None] > torch.arange(n - ql, n, device="cuda")[:, None], float("-inf"))
        want.append(torch.einsum("hqk,khd->qhd", x.softmax(-1), kv[s:s + n, :, dim:].double()))
    assert _rel(out, torch.cat(want)) < LIMIT[split, out.dtype], _rel(out, torch.cat(want))


@pytest.mark.parametrize("lens", [None, [5, 130, 64]])
def test_gathered_rows_end_in_zeros(lens):
    cache = torch.randn(12, 64, 72, device="cuda", dtype=torch.bfloat16)
    bt = torch.arange(1, 12, dtype=torch.int32, device="cuda")[:9].view(3, 3).contiguous()
    starts = [0, 128, 320, 384] if lens else [0, 5, 135, 199]
    got = torch.full((starts[-1], 72), float("nan"), device="cuda", dtype=torch.bfloat16)
    cu().gather_cache(cache, bt, torch.tensor(starts, dtype=torch.int32, device="cuda"), got, 192,
                      lens=None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda"))
    want = torch.zeros_like(got)
    for i, n in enumerate(lens or [5, 130, 64]):
        want[starts[i]:starts[i] + n] = cache[bt[i].long()].view(-1, 72)[:n]
    assert torch.equal(got, want)


@pytest.mark.parametrize("H,R,P", [(16, 512, 64), (32, 512, 64), (5, 136, 16), (128, 512, 64)])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("splits", [1, 3])
def test_latent_rows(H, R, P, wide, splits):
    lens = [1, 63, 64, 65, 200, 1030]
    g = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    cache, q, qp = rnd(60, 64, R + P), rnd(len(lens), H, R), rnd(len(lens), H, P)
    bt = torch.randperm(60, device="cuda", generator=g)[:17].int()[None].repeat(len(lens), 1).contiguous()
    got = cu().mla_decode_tc(q, qp, cache, bt, torch.tensor(lens, dtype=torch.int32, device="cuda"), 0.06, max(lens), splits, wide=wide)
    cu().check_kernel_error(q.device)
    want = []
    for i, n in enumerate(lens):
        kv = cache[bt[i].long()].view(-1, R + P)[:n].double()
        w = (torch.cat([q[i], qp[i]], -1).double() @ kv.t() * 0.06).softmax(-1)
        want.append(w @ kv[:, :R])
    assert _rel(got, torch.stack(want)) < LIMIT[wide, got.dtype], _rel(got, torch.stack(want))
