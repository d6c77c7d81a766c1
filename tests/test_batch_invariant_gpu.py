"""VLLM_BATCH_INVARIANT=1: bits of the same rows alone and inside batches above every threshold of the default dispatch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _mode(monkeypatch):
    from vllm_b200 import envs
    from vllm_b200.ops import cuda as cu
    monkeypatch.setenv("VLLM_BATCH_INVARIANT", "1")
    envs._cache.clear()
    envs.disable_envs_cache()
    cu._plan_cache.clear()
    cu._fp8_plan_cache.clear()
    yield
    envs._cache.clear()
    cu._plan_cache.clear()
    cu._fp8_plan_cache.clear()


def _rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("H", [1024, 2048, 4096, 8192])
@pytest.mark.parametrize("gemma", [False, True])
def test_norms(H, gemma):
    from vllm_b200.ops import cuda as cu
    big, n, k = 1300, 300, 3                                       # more threads per row than rows leave, below and above 1024 rows
    x, r, y = _rnd(big, H), _rnd(big, H, seed=1), _rnd(big * k, H, seed=2)
    w, v = _rnd(H, seed=3), _rnd(H, seed=4)
    inv = torch.arange(big * k, dtype=torch.int32, device="cuda")
    tw = torch.rand(big, k, device="cuda")
    runs = {"norm": lambda m: (cu.rms_norm(x[:m], w, 1e-6, gemma),),
            "add": lambda m: cu.fused_add_rms_norm(x[:m].clone(), r[:m].clone(), w, 1e-6, gemma),
            "tail": lambda m: cu.norm_add_norm(x[:m], r[:m].clone(), w, 1e-6, v, 1e-5, gemma),
            "experts": lambda m: cu.moe_combine_norm(y[:m * k], inv[:m * k], tw[:m], r[:m].clone(), w, 1e-6, gemma, x[:m])}
    for name, run in runs.items():
        for a, b in zip(run(n), run(big)):
            assert torch.equal(a, b[:n]), name


@pytest.mark.parametrize("Hq,Hkv,window,cap", [(32, 8, None, 0.0), (32, 8, 100, 0.0), (16, 4, None, 50.0), (8, 2, None, 1.0), (32, 8, 129, 50.0)])
def test_prompt_attention(Hq, Hkv, window, cap):
    """A prompt of 300 tokens alone, in portions, in a captured step's form, and in front of 12000 other tokens."""
    import dataclasses
    from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout
    from vllm_b200.ops import cuda as cu
    lens = [300] + [3000] * 4
    q, cache, md = _mk_attn_case(len(lens), Hq, Hkv, 128, 64, lens, lens)
    q, cache, md.kv_vt = q * 2, _to_tc_layout(cache), True
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731

    def portion(a, b, **kw):
        one = dataclasses.replace(md, num_reqs=1, num_actual_tokens=b - a, max_query_len=b - a, max_seq_len=b, query_start_loc=i32(0, b - a),
                                  seq_lens=i32(b), block_table=md.block_table[:1], **kw)
        return cu.paged_attention(q[a:b], cache, one, 0.1, window, cap)
    want = cu.paged_attention(q, cache, md, 0.1, window, cap)[:300]
    assert torch.equal(portion(0, 300), want)
    assert torch.equal(portion(0, 300, flat=True), want)
    assert torch.equal(torch.cat([portion(0, 77), portion(77, 205), portion(205, 206), portion(206, 300)]), want)


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("split", [False, True])
def test_expanded_prompts(window, split):
    from vllm_b200.ops import cuda as cu
    lens, H, D, V = [300] + [3000] * 4, 16, 64, 64
    T = sum(lens)
    q, k, v = _rnd(T, H, D, seed=5), _rnd(T, H, D, seed=6), _rnd(T, H, V, seed=7)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731

    def run(n):
        m, out = sum(lens[:n]), torch.zeros(sum(lens[:n]), H, V, dtype=q.dtype, device="cuda")
        start = i32([sum(lens[:i]) for i in range(n)])
        cu.mla_prefill(q[:m], k[:m], v[:m], out, start, i32(lens[:n]), i32(lens[:n]), start, 0, max(lens[:n]), 0.1, window=window, split=split)
        return out[:300]
    assert torch.equal(run(1), run(5))


@pytest.mark.parametrize("T,E,k", [(1200, 8, 4), (2100, 64, 8), (600, 4, 2)])
def test_experts(T, E, k):
    """A few tokens alone and in a batch above 1024 pairs and above 64 pairs for each expert."""
    from vllm_b200.ops import moe
    H, inter = 2048, 192
    x, w13, w2 = _rnd(T, H), _rnd(E, 2 * inter, H, seed=1, scale=H ** -0.5), _rnd(E, H, inter, seed=2, scale=inter ** -0.5)
    g = torch.Generator(device="cuda").manual_seed(3)
    ids = torch.rand(T, E, device="cuda", generator=g).topk(k, -1).indices.int()
    w = torch.rand(T, k, device="cuda", generator=g)
    whole = moe.fused_moe_cuda(x, w13, w2, w, ids)
    for n in (1, 30, 250):
        assert torch.equal(moe.fused_moe_cuda(x[:n].contiguous(), w13, w2, w[:n].contiguous(), ids[:n].contiguous()), whole[:n])


def test_block_scaled_products():
    from vllm_b200.ops import cuda as cu, ref
    x = _rnd(2000, 512)
    wq, ws = ref.block_quant_weight_fp8(torch.randn(8192, 512, device="cuda") * 0.05, 128)
    xq, xs = cu.per_token_group_quant_fp8(x, 128, col_major=True)
    whole = cu.gemm_fp8_block(xq, xs, wq, ws.contiguous())
    xq, xs = cu.per_token_group_quant_fp8(x[:200].contiguous(), 128, col_major=True)
    assert torch.equal(cu.gemm_fp8_block(xq, xs, wq, ws.contiguous()), whole[:200])
