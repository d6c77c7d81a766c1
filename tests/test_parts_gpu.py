"""Several linear layers of one input in one launch, and router logits read in 16 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 17, 24, 128])
@pytest.mark.parametrize("K,parts", [(2048, [(1536, "silu", False), (32, None, False), (1, None, False)]), (1024, [(1024, 128, False), (256, None, True), (255, None, True)]),
                                     (192, [(12, "silu", False), (129, None, True)]), (64, [(8, 4, True), (8, None, False), (1000, None, False), (16640, None, False)])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_products_of_one_input(M, K, parts, dtype):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(M + K)
    wide = torch.randn(M, K + 8, device="cuda", generator=g).to(dtype)
    x = wide[:, :K]                                                    # rows at a stride of their own
    ws = [(torch.randn(n, K, device="cuda", generator=g) * K ** -0.5).to(dtype) for n, _, _ in parts]
    bs = [torch.randn(n, device="cuda", generator=g).to(dtype) if b else None for n, _, b in parts]
    forms = [f for _, f, _ in parts]
    got = cu.linear_parts(x, ws, bs, forms)
    assert (got is None) == (sum(-(-n // 128) for n, _, _ in parts) > cu.PARTS_TILES)
    if got is None:
        return
    u, tiny = (2.0 ** -8, 0.0) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    for y, w, b, f in zip(got, ws, bs, forms):
        exact = x.double() @ w.double().T
        bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)       # of the sums in 32 bits, in any order
        if b is not None:
            exact, bound = exact + b.double(), bound + 2.0 ** -24 * b.double().abs()
        if f == "silu":
            gate, up = exact[:, ::2], exact[:, 1::2]
            want = gate * torch.sigmoid(gate) * up
            # |silu'| <= 1.1, |silu(g)| <= |g|; a quick exponential and division: a few 2^-22
            bound = 1.1 * bound[:, ::2] * up.abs() + gate.abs() * bound[:, 1::2] + 1.1 * bound[:, ::2] * bound[:, 1::2] + 2.0 ** -20 * (gate * up).abs()
        elif f:
            want, bound = (t.view(M, -1, 2, f).transpose(0, 2).transpose(1, 2).reshape(2, M, -1) for t in (exact, bound))
        else:
            want = exact
        assert y.shape == want.shape and y.dtype == dtype and y.is_contiguous()
        assert bool(((y.double() - want).abs() <= bound * (1 + u) + u * want.abs() + tiny).all())


def test_rows_and_forms_that_are_not_covered():
    from vllm_b200.ops import cuda as cu
    x, w = torch.zeros(129, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16)
    assert cu.linear_parts(x, [w, w], [None] * 2, [None] * 2) is None
    assert cu.linear_parts(x[:4], [w], [None], [None]) is None and cu.linear_parts(x[:4], [w] * 5, [None] * 5, [None] * 5) is None
    assert cu.linear_parts(x[:4].float(), [w, w], [None] * 2, [None] * 2) is None and cu.linear_parts(x[:4], [w, w.half()], [None] * 2, [None] * 2) is None
    assert cu.linear_parts(x[:4], [w, w[:, :32]], [None] * 2, [None] * 2) is None and cu.linear_parts(x[:4], [w, w], [None] * 2, [None, 6]) is None
    assert cu.linear_parts(x[:0], [w, w], [None] * 2, [None] * 2) is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scoring", ["sigmoid", "softmax"])
def test_router_logits_in_16_bits(dtype, scoring):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(3)
    lg = torch.randn(37, 32, device="cuda", generator=g).to(dtype)
    bias = torch.randn(32, device="cuda", generator=g)
    a, b = (cu.grouped_topk(t, 6, 4, 2, True, scoring, bias, 2.5) for t in (lg, lg.float()))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("E,groups,keep,k", [(32, 4, 2, 6), (33, 1, 1, 33 - 1), (64, 8, 3, 8), (96, 32, 32, 32), (160, 5, 2, 7), (256, 8, 4, 8), (256, 1, 1, 1), (24, 3, 1, 8)])
@pytest.mark.parametrize("scoring,biased,top2", [("sigmoid", True, "top2"), ("softmax", False, "max"), ("sigmoid", True, "max")])
def test_a_warp_per_token_chooses_as_a_block(E, groups, keep, k, scoring, biased, top2):
    """Equal scores (the first expert wins), infinities and NaN among them; the block form takes the same numbers behind a router of its own: an identity."""
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(E + k)
    lg = torch.randint(-4, 5, (1101, E), device="cuda", generator=g).float() / 2
    lg[::7] = torch.randn(lg[::7].shape, device="cuda", generator=g)
    lg[3, ::3], lg[5, 1] = float("-inf"), float("inf") if scoring == "sigmoid" else 50.0
    bias = torch.randint(-2, 3, (E,), device="cuda", generator=g).float() if biased else None
    a = cu.grouped_topk(lg, k, groups, keep, True, scoring, bias, 2.5, top2)
    s = lg.double().sigmoid() if scoring == "sigmoid" else lg.double().softmax(-1)
    s32 = lg.sigmoid() if scoring == "sigmoid" else s.float()
    for t in (0, 3, 5, 7, *range(100, 1101, 91)):
        ch = (s32[t] + (bias if biased else 0)).view(groups, -1)
        gs = ch.topk(2, -1).values.sum(-1) if top2 == "top2" and E // groups > 1 else ch.max(-1).values
        ids = a[1][t].long()
        n = min(k, keep * (E // groups))
        assert len(set(ids[:n].tolist())) == n
        kept = set((ids[:n] // (E // groups)).tolist())
        eps = 4e-7 * (1 + float(ch.abs().max()))                  # scores in 32 bits on both sides
        assert len(kept) <= keep
        if groups > 1:
            out = [i for i in range(groups) if i not in kept]
            full = [i for i in kept]
            if len(kept) == keep and out:
                assert float(gs[full].min()) >= float(gs[out].max()) - 2 * eps
        inside = torch.zeros(groups, device="cuda", dtype=torch.bool)
        inside[list(kept)] = True
        c = torch.where(inside[:, None].expand(ch.shape), ch, torch.full_like(ch, float("-inf"))).view(-1)
        picked = c[ids[:n]]
        assert bool((picked[:-1] >= picked[1:] - eps).all())
        rest = c.clone()
        rest[ids[:n]] = float("-inf")
        if len(kept) == keep:
            assert float(picked[-1]) >= float(rest.max()) - eps
        w = s[t, ids[:n]]
        want = w * 2.5 / s32[t, ids].sum().double()
        assert torch.allclose(a[0][t, :n].double(), want, rtol=1e-5, atol=1e-12)


@pytest.mark.parametrize("E,k", [(1, 1), (8, 2), (32, 32), (33, 4), (64, 8), (129, 6), (512, 32)])
@pytest.mark.parametrize("renorm", [False, True])
def test_softmax_router(E, k, renorm):
    """Equal logits (the first expert wins), a row whose other experts round to nothing, one with NaN."""
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(E)
    lg = torch.randint(-3, 4, (70, E), device="cuda", generator=g).float()
    lg[1] = -200.0
    lg[1, E // 2] = 0.0
    w, ids = cu.topk_softmax(lg, k, renorm)
    want = lg.double().softmax(-1)
    order = lg.sort(dim=-1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(ids.long(), order)
    p = want.gather(1, order)
    p = p / p.sum(-1, keepdim=True) if renorm else p
    # a quick exponential (2^-21 of it and 2^-23 of its argument, at most 6 here) and sums of up to 512 numbers in 32 bits
    assert torch.allclose(w.double(), p, rtol=2.0 ** -17, atol=1e-30)
    if E > 1:
        lg[2, 0] = float("nan")
        assert int(cu.topk_softmax(lg, 1, renorm)[1][2]) != 0
