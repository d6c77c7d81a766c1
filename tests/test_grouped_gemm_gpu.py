"""Grouped GEMM of prompt-sized expert batches: edges of tiles, empty experts, gated activations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("rows,N,K", [([0, 1, 127, 128, 129, 0, 300], 512, 256), ([640], 208, 72), ([5, 700] * 20, 96, 1032),
                                      ([257, 0, 0, 90], 1040, 64)])
@pytest.mark.parametrize("act", [None, "silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_grouped_rows(rows, N, K, act, dtype):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(1)
    R, E = sum(rows), len(rows)
    x = torch.randn(R, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(E, N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    offs = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device="cuda")
    got = cu.gemm_grouped(x, w, offs, act)
    cu.check_kernel_error(x.device)
    fn = {"silu": torch.nn.functional.silu, "gelu": torch.nn.functional.gelu,
          "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh")}
    want = []
    for xe, we in zip(x.split(rows), w):
        h = xe.double() @ we.double().t()
        want.append(h if act is None else fn[act](h[:, :N // 2]) * h[:, N // 2:])
    # one rounding of the result: at most 2^-8 (bf16) or 2^-11 (fp16) of each value, 2^-9.35 or 2^-12.35 in the 2-norm (test_prompt_attention_gpu.py)
    assert _rel(got, torch.cat(want)) < (2 ** -9 if dtype == torch.bfloat16 else 2 ** -12)


@pytest.mark.parametrize("rows,N,K", [([0, 1, 255, 256, 257, 300, 129, 0], 512, 256), ([700], 208, 72), ([130] * 40, 96, 1032), ([2999, 1], 1040, 64)])
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_of_pairs_of_blocks(rows, N, K, act, dtype):
    """Sizes that go to pairs of blocks: edges of their 256 rows, a second block without rows, more tiles than pairs."""
    test_grouped_rows(rows, N, K, act, dtype)


@pytest.mark.parametrize("T,E,k", [(300, 8, 4), (600, 4, 2), (2100, 64, 8)])
@pytest.mark.parametrize("mapped", [False, True])
def test_prompt_experts_match_decode_experts(T, E, k, mapped):
    """The device path of large batches against the one of small batches, a few tokens at a time."""
    from vllm_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(2)
    H, inter = 256, 192
    rnd = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)  # noqa: E731
    x, w13, w2 = rnd(T, H), rnd(E, 2 * inter, H, scale=H ** -0.5), rnd(E, H, inter, scale=inter ** -0.5)
    ids = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices.int()
    w = torch.rand(T, k, device="cuda", generator=g)
    emap = None
    if mapped:                                  # experts of other ranks are dropped
        emap = torch.full((2 * E,), -1, dtype=torch.int32, device="cuda")
        emap[E // 2:E // 2 + E] = torch.arange(E, dtype=torch.int32, device="cuda")
        ids = ids + (torch.arange(T, device="cuda") % 3 == 0).int()[:, None] * (E // 2)
    got = moe.fused_moe_cuda(x, w13, w2, w, ids, "silu", emap)
    n = moe.GROUPED_MAX_ROWS // k
    want = torch.cat([moe.fused_moe_cuda(x[i:i + n], w13, w2, w[i:i + n], ids[i:i + n], "silu", emap) for i in range(0, T, n)])
    assert _rel(got, want) < 2 ** -7            # hidden rows rounded to bf16 on one side only, and both results


@pytest.mark.parametrize("R,E,bn", [(6, 32, 16), (144, 32, 16), (384, 32, 32), (256, 16, 32), (513, 64, 32), (1000, 128, 16), (40, 8, 16)])
def test_both_grids_of_decode_experts(R, E, bn):
    """Grid by rows and grid by possible chunks: the same products, also where most experts have no row and rows are missing at the end."""
    from vllm_b200.ops import cuda as cu, moe
    assert moe.flat_grid(R, E, bn) == (bn == 16 or E * -(-R // bn) > 128)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(R, 128, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(E, 136, 128, device="cuda", generator=g).to(torch.bfloat16)
    for spread in (E, max(E // 8, 1)):
        n = torch.bincount(torch.randint(0, spread, (R - R // 10,), device="cuda", generator=g) * (E // spread), minlength=E)
        offs = torch.cat([n.new_zeros(1), n.cumsum(0)]).int()
        a, b = (cu.gemm_tc_grouped(x, w, offs, bn, flat=f)[:R - R // 10] for f in (False, True))
        assert torch.equal(a, b)
        want = torch.cat([xe.double() @ we.double().t() for xe, we in zip(x[:R - R // 10].split(n.tolist()), w)])
        assert _rel(a, want) < 2 ** -9


@pytest.mark.parametrize("E,act", [(1024, "silu"), (600, "gelu_tanh"), (512, "silu")])
def test_more_experts_than_the_prompt_tiles_take(E, act):
    """64 pairs for each of more than 512 experts: the decode tiles go on with them."""
    from vllm_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(torch.bfloat16)  # noqa: E731
    T, k, H, inter = 8 * E, 8, 64, 64
    x, w13, w2 = rnd(T, H), rnd(E, 2 * inter, H, scale=H ** -0.5), rnd(E, H, inter, scale=inter ** -0.5)
    ids = (torch.arange(T * k, device="cuda").view(T, k) * 7 % E).int()
    w = torch.rand(T, k, device="cuda", generator=g)
    got = moe.fused_moe_rows(x, w13, w2, w, ids, act, None, True)
    n = 100
    want = moe.fused_moe_rows(x[:n], w13, w2, w[:n], ids[:n], act, None, True)
    assert _rel(got[:n], want) < 2 ** -7            # hidden rows rounded to bf16 on one side only, and both results


def test_refused_activations_are_refused_at_every_size():
    from vllm_b200.ops import moe
    x = torch.zeros(300, 64, device="cuda", dtype=torch.bfloat16)
    w13, w2 = torch.zeros(4, 128, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(4, 64, 64, device="cuda", dtype=torch.bfloat16)
    ids, w = torch.arange(1200, device="cuda").view(300, 4).int() % 4, torch.ones(300, 4, device="cuda")
    for n in (10, 300):
        with pytest.raises(KeyError):
            moe.fused_moe_cuda(x[:n], w13, w2, w[:n], ids[:n], "swish")
