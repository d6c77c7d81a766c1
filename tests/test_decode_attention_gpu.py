"""Decode attention on 64-token pages against 64 bits: parts of the keys, edges of pages and of a warp's 16 tokens, windows, sinks, foreign slots."""
import pytest
import torch

from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout, cu

pytestmark = pytest.mark.gpu
LENS = [1, 15, 16, 17, 63, 64, 65, 128, 300, 1030]


def _exact(q, cache, bt, lens, scale, window, cap, chunk, sinks):
    """Result, its log-sum-exp and the sum of p |v|, all of 64 bits."""
    B, Hq, D = q.shape
    Hkv = cache.shape[2]
    out, mass, lse = (torch.zeros(B, Hq, n, dtype=torch.float64, device="cuda") for n in (D, D, 1))
    for b, n in enumerate(lens):
        blocks = bt[b, :-(-n // 64)].long()
        k = cache[blocks, 0].double().transpose(1, 2).reshape(-1, Hkv, D)[:n].repeat_interleave(Hq // Hkv, 1)
        v = cache[blocks, 1].double().transpose(1, 2).reshape(-1, Hkv, D)[:n].repeat_interleave(Hq // Hkv, 1)
        s = torch.einsum("hd,nhd->hn", q[b].double(), k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        first = max(n - window if window else 0, (n - 1) // chunk * chunk if chunk else 0, 0)
        s[:, :first] = float("-inf")
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        lse[b, :, 0] = torch.logsumexp(s, -1)
        w = s.softmax(-1)[:, :n]
        out[b], mass[b] = torch.einsum("hn,nhd->hd", w, v), torch.einsum("hn,nhd->hd", w, v.abs())
    return out, mass, lse[..., 0]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (4, 2), (12, 3), (16, 2), (16, 1)])
@pytest.mark.parametrize("parts,window,chunk,cap,sink", [(0, None, 0, 0.0, False), (1, None, 0, 0.0, True), (2, 100, 0, 0.0, False), (3, None, 0, 30.0, False),
                                                         (5, 16, 0, 30.0, True), (16, None, 0, 0.0, True), (2, None, 128, 0.0, False), (0, 512, 0, 0.0, False)])
def test_against_64_bits(dtype, Hq, Hkv, parts, window, chunk, cap, sink):
    B = len(LENS)
    q, cache, md = _mk_attn_case(B, Hq, Hkv, 128, 64, LENS, [1] * B, dtype=dtype, seed=Hq + parts)
    q = q * 4
    sinks = torch.randn(Hq, device="cuda") if sink else None
    want, mass, lse = _exact(q, cache, md.block_table, LENS, 128 ** -0.5, window, cap, chunk, sinks)
    for b, n in enumerate(LENS):                     # what lies behind a sequence, or in front of its window, is another's
        last = int(md.block_table[b, (n - 1) // 64])
        cache[last, :, :, (n - 1) % 64 + 1:] = float("nan")
        if window and n > window:
            for t in range(n - window):
                cache[int(md.block_table[b, t // 64]), :, :, t % 64] = float("inf")
    md.kv_vt, md.num_splits = True, parts
    got, got_lse = cu().paged_attention(q, _to_tc_layout(cache), md, 128 ** -0.5, sliding_window=window, logits_soft_cap=cap, chunk_size=chunk,
                                        sinks=sinks, return_lse=True)
    # weights are held in two parts of 16 bits, the result is rounded once; 32-bit sums and exponentials beside them
    u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11         # half a unit in the last place of 8 and 11 bits, at worst
    bound = u * u * mass + u * want.abs() + 4e-5 * mass + (6e-8 if dtype is torch.float16 else 0.0)
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() / bound).max()
    assert (got_lse.double() - lse).abs().max() < 2e-4
    again = cu().paged_attention(q, _to_tc_layout(cache), md, 128 ** -0.5, sliding_window=window, logits_soft_cap=cap, chunk_size=chunk, sinks=sinks)
    assert torch.equal(again, got)


@pytest.mark.parametrize("copies,parts", [(1, 1), (16, 1), (16, 3), (48, 1), (24, 2)])
def test_forms(copies, parts):
    """CTAs per SM and pages on their way go by the number of CTAs."""
    lens = LENS * copies
    q, cache, md = _mk_attn_case(len(lens), 8, 2, 128, 64, lens, [1] * len(lens), seed=copies)
    want, mass, _ = _exact(q, cache, md.block_table, lens, 0.09, None, 0.0, 0, None)
    md.kv_vt, md.num_splits = True, parts
    got = cu().paged_attention(q, _to_tc_layout(cache), md, 0.09)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -16 + 4e-5) * mass).all()


def test_rules():
    c = cu()
    n = c.num_sms()
    assert [c.decode_form(x) for x in (1, n, n + 1, 6 * n, 6 * n + 1)] == [0, 0, 1, 1, 2]
    assert c.decode_parts(n, 1, 4096) == 1 and c.decode_parts(1, 2, 64) == 1 and c.decode_parts(1, 2, 4096) == 8
    for B, Hkv, k in ((1, 1, 1), (1, 8, 130), (64, 4, 4096), (1, 1, 1 << 17), (1000, 8, 4096)):
        p = c.decode_parts(B, Hkv, k)
        assert p in (1, 2, 4, 8) and (p == 1 or B * Hkv * p <= n)
