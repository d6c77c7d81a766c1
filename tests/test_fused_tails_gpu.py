"""Block tails in one pass (norm + add + norm; expert combine + shared expert + add + norm) and values turned into transposed pages."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rel(x, y):
    return float((x.double() - y).norm() / y.norm())


def _norm(x, w, gemma, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * (w + 1 if gemma else w)


@pytest.mark.parametrize("T,H", [(1, 64), (3, 2048), (700, 1032), (5, 16384), (1025, 2056), (1024, 8192)])
@pytest.mark.parametrize("gemma", [False, True])
@pytest.mark.parametrize("dtype", [BF, torch.float16])
def test_norm_add_norm(T, H, gemma, dtype):
    from vllm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    x, r = (torch.randn(T, H, device="cuda", generator=g).to(dtype) for _ in range(2))
    w1, w2 = ((torch.randn(H, device="cuda", generator=g) * 0.1 + (0 if gemma else 1)).to(dtype) for _ in range(2))
    s = r.double() + _norm(x.double(), w1.double(), gemma, 1e-6)
    y, r2 = ops.norm_add_norm(x, r, w1, 1e-6, w2, 1e-5, gemma)
    ulp = 2 ** -9 if dtype == BF else 2 ** -12               # above the 2^-9.35 and 2^-12.35 of a rounding in the 2-norm (test_prompt_attention_gpu.py)
    assert r2 is r and _rel(r, s) < ulp                      # one rounding
    assert _rel(y, _norm(s, w2.double(), gemma, 1e-5)) < 2 * ulp          # of the stream, and its own


@pytest.mark.parametrize("T,H,k", [(1, 64, 1), (37, 2048, 6), (300, 1032, 3), (2, 9000, 2), (9, 2048, 9)])
@pytest.mark.parametrize("shared", [None, "plain", "gated"])
def test_combine_norm(T, H, k, shared):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    rows, r, nw = rnd(T * k, H).to(BF), rnd(T, H).to(BF), (1 + 0.1 * rnd(H)).to(BF)
    inv = torch.randperm(T * k, device="cuda", generator=g).int()
    inv[torch.rand(T * k, device="cuda", generator=g) < 0.2] = -1          # pairs of other ranks
    w = torch.rand(T, k, device="cuda", generator=g)
    extra = None if shared is None else rnd(T, H).to(BF)
    gate = rnd(T, 1).to(BF) if shared == "gated" else None
    picked = rows.double()[inv.clamp_min(0).long()] * (inv >= 0)[:, None]
    s = r.double() + (picked.view(T, k, H) * w.double()[..., None]).sum(1)
    if extra is not None:
        s = s + extra.double() * (1 if gate is None else gate.double().sigmoid())
    y, r2 = cu.moe_combine_norm(rows, inv, w, r, nw, 1e-6, False, extra, gate)
    assert r2 is r and _rel(r, s) < 2 ** -9
    assert _rel(y, _norm(s, nw.double(), False, 1e-6)) < 2 ** -8


@pytest.mark.parametrize("Hkv,D,BS", [(2, 128, 64), (1, 64, 16), (3, 128, 32), (1, 256, 64), (2, 128, 4)])
def test_values_turned(Hkv, D, BS):
    """Slots that follow one another from any place, gaps, padding, shuffled ones; both kernels that use it."""
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(3)
    runs = [list(range(3, 70)), list(range(BS * 20, BS * 20 + 130)), [-1] * 5, list(range(1000, 1007)), list(range(1016, 1024)), list(range(2001, 2100))]
    shuffled = (3000 + torch.randperm(60, generator=torch.Generator().manual_seed(1))).tolist()
    slots = torch.tensor(sum(runs, []) + shuffled, device="cuda")
    T = len(slots)
    assert T > 257
    qkv = torch.randn(T, (2 + 2 * Hkv) * D, device="cuda", generator=g).to(BF)
    q, k, v = qkv.split([2 * D, Hkv * D, Hkv * D], -1)
    cache = torch.zeros(-(-3100 // BS), 2, Hkv, BS, D, device="cuda", dtype=BF)
    pos, cs = torch.arange(T, device="cuda") % 50, torch.randn(50, D, device="cuda", generator=g)
    want = torch.zeros_like(cache[:, 1]).view(-1, Hkv, D, BS)
    for t, s in enumerate(slots.tolist()):
        if s >= 0:
            want[s // BS, :, :, s % BS] = v[t].view(Hkv, D)
    cu.rope_and_cache(pos, q, k, v, cs, D, True, cache, slots, vt=True)
    assert torch.equal(cache[:, 1].reshape(want.shape), want)
    if cu.qknorm_rope_ok(D, D, True):
        cache.zero_()
        w = torch.ones(D, device="cuda", dtype=BF)
        cu.fused_qk_norm_rope(pos, q, k, w, w, cs, D, 1e-6, True, v=v, kv_cache=cache, slot_mapping=slots, vt=True)
        assert torch.equal(cache[:, 1].reshape(want.shape), want)


@pytest.mark.parametrize("T,H", [(1024, 2048), (1030, 2056), (1024, 16384), (1023, 2048)])
@pytest.mark.parametrize("add", [False, True])
def test_norms_of_prompts(T, H, add):
    """Rows whose threads take several vectors, and the last batch that takes one."""
    from vllm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(4)
    x, r, w = (torch.randn(*s, device="cuda", generator=g).to(BF) for s in ((T, H), (T, H), (H,)))
    s = (x.float() + r.float()).to(BF) if add else x.clone()
    y = ops.fused_add_rms_norm(x, r, w, 1e-6)[0] if add else ops.rms_norm(x, w, 1e-6)
    assert not add or torch.equal(r, s)
    assert _rel(y, _norm(s.double(), w.double(), False, 1e-6)) < 2 ** -9
