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
    # weights are held in 16 bits, those of capped scores in two parts of 16; the result is rounded once; 32-bit sums and exponentials beside them
    u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11         # half a unit in the last place of 8 and 11 bits, at worst
    bound = (u * u if cap else u) * mass + u * want.abs() + 4e-5 * mass + (6e-8 if dtype is torch.float16 else 0.0)
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() / bound).max()
    assert (got_lse.double() - lse).abs().max() < 2e-4
    again = cu().paged_attention(q, _to_tc_layout(cache), md, 128 ** -0.5, sliding_window=window, logits_soft_cap=cap, chunk_size=chunk, sinks=sinks)
    assert torch.equal(again, got)


@pytest.mark.parametrize("copies,parts", [(1, 1), (16, 1), (16, 3), (48, 1), (24, 2)])
def test_forms(copies, parts):
    """Many requests and few, in one part and in several."""
    lens = LENS * copies
    q, cache, md = _mk_attn_case(len(lens), 8, 2, 128, 64, lens, [1] * len(lens), seed=copies)
    want, mass, _ = _exact(q, cache, md.block_table, lens, 0.09, None, 0.0, 0, None)
    md.kv_vt, md.num_splits = True, parts
    got = cu().paged_attention(q, _to_tc_layout(cache), md, 0.09)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -8 + 4e-5) * mass).all()


@pytest.mark.parametrize("R,P,dtype", [(512, 64, torch.bfloat16), (512, 64, torch.float16), (512, 0, torch.bfloat16), (384, 64, torch.bfloat16),
                                       (72, 40, torch.bfloat16), (192, 16, torch.bfloat16)])
@pytest.mark.parametrize("H,BS", [(1, 64), (16, 64), (17, 16), (40, 128)])
@pytest.mark.parametrize("parts,window,wide", [(0, None, False), (1, 100, True), (3, None, True), (16, 16, False)])
def test_latents_against_64_bits(R, P, dtype, H, BS, parts, window, wide):
    g = torch.Generator(device="cuda").manual_seed(R + H)
    B, mb = len(LENS), -(-max(LENS) // BS)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)                    # noqa: E731
    q, qp, cache = rnd(B, H, R), rnd(B, H, P) if P else None, rnd(B * mb + 1, BS, R + P)
    bt = (torch.randperm(B * mb, device="cuda", generator=g) + 1).int().view(B, mb)
    scale = 3.0 / (R + P) ** 0.5
    want, mass = (torch.zeros(B, H, R, dtype=torch.float64, device="cuda") for _ in range(2))
    lse = torch.zeros(B, H, dtype=torch.float64, device="cuda")
    bad = cache.clone()
    for b, n in enumerate(LENS):
        rows = cache[bt[b].long()].view(-1, R + P)[:n].double()
        first = max(0, n - window) if window else 0
        s = (torch.cat([q[b], qp[b]], -1) if P else q[b]).double() @ rows[first:].t() * scale
        w, lse[b] = s.softmax(-1), torch.logsumexp(s, -1)
        want[b], mass[b] = w @ rows[first:, :R], w @ rows[first:, :R].abs()
        for t in [*range(first), *range(n, mb * BS)]:
            bad[int(bt[b, t // BS]), t % BS] = float("nan")
    got, got_lse = cu().mla_decode_tc(q, qp, bad, bt, torch.tensor(LENS, dtype=torch.int32, device="cuda"), scale, max(LENS), parts, return_lse=True,
                                      sliding_window=window, wide=wide)
    # weights of 16 bits or (wide) in two parts of 16, the result rounded once; 32-bit sums and exponentials of scores up to 16 beside them
    u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    bound = (u * u if wide else u) * mass + u * want.abs() + 4e-5 * mass + (6e-8 if dtype is torch.float16 else 0.0)
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() / bound).max()
    assert (got_lse.double() - lse).abs().max() < 2e-4
