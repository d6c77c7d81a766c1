"""What a kernel for some sizes or some company computes is, bit for bit, what the kernel for the others computes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 24, 64, 100, 128])
@pytest.mark.parametrize("K,parts", [(2048, [(1536, "silu", False), (32, None, False), (1, None, False)]), (2048, [(4096, 128, False), (512, None, False), (512, None, True)]),
                                     (1024, [(2048, 64, True), (256, None, True), (255, None, True), (8, None, False)]), (2048, [(1024, None, False), (576, None, False)]),
                                     (576, [(4992, None, True), (128, "silu", False)]), (4096, [(128, None, False), (13000, None, False)])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_products_together_and_alone(M, K, parts, dtype):
    """Products that share a launch add their partial sums as each does alone: more and fewer CTAs of a cluster than a matrix has sums."""
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    ws = [(torch.randn(n, K, device="cuda", generator=g) * K ** -0.5).to(dtype) for n, _, _ in parts]
    bs = [torch.randn(n, device="cuda", generator=g).to(dtype) if b else None for n, _, b in parts]
    got = cu.linear_parts(x, ws, bs, [f for _, f, _ in parts])
    assert got is not None or (M > 64 and len(parts) == 2 and K == 4096)         # (there no cluster holds the sums of 103 tiles)
    for y, w, b, (n, f, _) in zip(got or [], ws, bs, parts):
        alone = cu.gemm_tc(x, w, b, act=int(f == "silu"))
        if isinstance(f, int):
            alone = alone.view(M, -1, 2, f).permute(2, 0, 1, 3).reshape(2, M, -1)
        assert torch.equal(y, alone)


@pytest.mark.parametrize("R,I,K,E", [(48, 512, 1024, 16), (144, 768, 2048, 32), (7, 64, 192, 300), (300, 128, 64, 2), (1000, 192, 128, 9)])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_experts_streamed_and_by_tiles(R, I, K, E, act, dtype):
    """Hidden rows and outputs of a few rows per expert are those of the product by tiles with the activation behind it."""
    from vllm_b200.ops import cuda as cu
    from vllm_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(R + E)
    x = torch.randn(R, K, device="cuda", generator=g).to(dtype)
    w13 = (torch.randn(E, 2 * I, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    w2 = (torch.randn(E, K, I, device="cuda", generator=g) * I ** -0.5).to(dtype)
    ids = torch.randint(0, E, (R, 1), device="cuda", generator=g, dtype=torch.int32)
    tok, inv, offs = cu.moe_align(ids, E)
    xs, bn = cu.moe_gather(x, tok), moe._tile_width(R, E)
    want = cu.act_and_mul(cu.gemm_tc_grouped(xs, w13, offs, bn), act)
    for width in (16, 32, 64, 128):
        assert torch.equal(cu.gemm_experts(xs, w13, offs, width, act, rounded=True), want)
    rows, where = moe.grouped_rows(x, w13, w2, ids, act, None)
    assert torch.equal(rows[where.long()], cu.gemm_tc_grouped(want, w2, offs, bn)[inv.long()])


@pytest.mark.parametrize("E,groups,keep", [(40, 1, 1), (64, 4, 3), (96, 4, 2), (128, 8, 4), (129, 3, 2), (160, 8, 3), (256, 1, 1), (256, 32, 8)])
@pytest.mark.parametrize("scoring,biased,top2", [("softmax", False, "max"), ("softmax", True, "top2"), ("sigmoid", True, "top2")])
@pytest.mark.parametrize("renorm", [False, True])
def test_router_of_few_and_many_tokens(E, groups, keep, scoring, biased, top2, renorm):
    """A warp per token and a block per token: by the number of tokens above 128 experts, by that of the choices (32 and 33) at all sizes."""
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(E + keep)
    lg = torch.randn(1100, E, device="cuda", generator=g) * 3
    bias = torch.randn(E, device="cuda", generator=g) * 0.1 if biased else None
    if biased:
        bias[1::5] = float("-inf")                   # experts that are never chosen
    lg[3, ::7], lg[4], lg[5, 2] = float("-inf"), float("-inf"), float("nan")
    if groups > 1:
        lg[6:9, :E // groups - 1] = float("-inf")    # one candidate in a group
    for t in (lg, lg.bfloat16()):
        few = [cu.grouped_topk(t[a:a + 100], 8, groups, keep, renorm, scoring, bias, 2.5, top2) for a in range(0, 1100, 100)]
        many = cu.grouped_topk(t, 8, groups, keep, renorm, scoring, bias, 2.5, top2)
        assert torch.equal(torch.cat([f[1] for f in few]), many[1])
        assert torch.equal(torch.cat([f[0] for f in few]).view(torch.int32), many[0].view(torch.int32))
        if E > 33:
            a, b = (cu.grouped_topk(t, k, groups, keep, False, scoring, bias, 1.0, top2) for k in (32, 33))
            assert torch.equal(a[1], b[1][:, :32]) and torch.equal(a[0].view(torch.int32), b[0][:, :32].contiguous().view(torch.int32))
