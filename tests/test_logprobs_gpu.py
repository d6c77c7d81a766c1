"""Log-probabilities of sampled and likeliest tokens: the kernel, and decode steps that replay the captured graph for them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,V,k", [(1, 7, 7), (3, 1000, 0), (5, 32000, 5), (2, 50257, 20), (64, 1024, 1), (2, 128256, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_kernel(B, V, k, dtype):
    from vllm_b200.ops import cuda as cu
    from vllm_b200.ops import ref
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(B, V, device="cuda", generator=g) * 4).to(dtype)
    x[0, V // 2] = float("-inf")
    sampled = torch.randint(0, V, (B,), device="cuda", generator=g)
    p = cu.logprobs(x, sampled, k)
    ids, vals, ranks = ref.compute_logprobs(x, sampled, k)
    assert torch.equal(p[:, 0].long(), sampled) and torch.equal(p[:, -1].long(), ranks)
    got = p[:, k + 1:2 * k + 2].contiguous().view(torch.float32)
    # 32-bit sums of V exponentials in another order
    assert float((got - vals).abs()[vals.isfinite()].max()) < 2e-5 * (1 + float(vals[vals.isfinite()].abs().max()))
    lp = x.float().log_softmax(-1)
    assert torch.allclose(lp.gather(1, p[:, 1:k + 1].long()), vals[:, 1:], atol=1e-4)           # ids may differ where values tie
    for row in p[:, 1:k + 1].tolist():
        assert len(set(row)) == len(row)


@pytest.mark.parametrize("extra", [dict(logprobs=3), dict(logprobs=0, temperature=0.9, seed=5), dict(logprobs=2, top_p=0.7, temperature=0.8, seed=1),
                                   dict(repetition_penalty=1.3), dict(top_k=5, temperature=1.0, seed=2), dict(logprobs=2, min_tokens=3)],
                         ids=["logprobs", "sampled", "top_p", "penalty", "top_k", "min_tokens"])
def test_captured_steps_match_eager_ones(extra):
    from vllm_b200 import LLM, SamplingParams
    prompts = [{"prompt_token_ids": [(7 * i + j) % 300 + 3 for j in range(5 + 3 * i)]} for i in range(5)]
    # one request without any of it in the same batch, one that ends early
    sp = [SamplingParams(**{**dict(temperature=0.0), **extra}, max_tokens=6 + i, ignore_eos=True) for i in range(4)]
    sp.append(SamplingParams(temperature=0.0, max_tokens=12, ignore_eos=True))
    got = []
    for eager in (True, False):
        llm = LLM("llama-small", max_model_len=256, max_num_seqs=8, max_num_batched_tokens=256, gpu_memory_utilization=0.2, load_format="dummy",
                  enforce_eager=eager, skip_tokenizer_init=True, dtype="bfloat16")
        runner = llm.llm_engine.engine_core.engine_core.model_executor.worker.runner
        got.append(llm.generate(prompts, sp))
        if not eager:
            assert sum(getattr(g, "replays", 0) for g in runner.graphs.values()) >= 8
        llm.shutdown()
    for a, b in zip(*got):
        a, b = a.outputs[0], b.outputs[0]
        assert list(a.token_ids) == list(b.token_ids)
        assert (a.logprobs is None) == (b.logprobs is None)
        for x, y in zip(a.logprobs or (), b.logprobs or ()):
            assert {t: v.rank for t, v in x.items()} == {t: v.rank for t, v in y.items()}
            for t in x:
                assert abs(x[t].logprob - y[t].logprob) < 1e-3


@pytest.mark.parametrize("V,k", [(33, 33), (8191, 64), (8193, 5), (8192, 8), (65536, 3), (65537, 20), (131073, 64), (262144, 1), (262145, 11)])       # around the ends of a CTA's and of a cluster's share
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_kernel_takes_ties_in_order_of_their_places(V, k, dtype):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randint(-3, 4, (3, V), device="cuda", generator=g).to(dtype)
    x[0, torch.randperm(V, device="cuda", generator=g)[:V - k // 2]] = float("-inf")        # fewer finite values than the list is long
    x[1, :V - 1] = -5                                                                       # the likeliest at the very end
    sampled = torch.tensor([0, V - 1, V // 2], device="cuda")
    p = cu.logprobs(x, sampled, k)
    order = x.float().sort(dim=-1, descending=True, stable=True)
    assert torch.equal(p[:, 1:k + 1].long(), order.indices[:, :k])
    assert torch.equal(p[:, -1].long(), (x > x.gather(1, sampled[:, None])).sum(-1) + 1)
    got = p[:, k + 1:2 * k + 2].contiguous().view(torch.float32).double()
    want = x.double().log_softmax(-1)
    want = torch.cat([want.gather(1, sampled[:, None]), want.gather(1, order.indices[:, :k])], 1)
    fin = want.isfinite()
    assert torch.equal(got.isfinite(), fin)
    # at most 13 additions of the sum follow one another in a share's tree of roundings after 32 in a thread, each 2^-24 of it; expf and logf a few more
    assert float((got - want).abs()[fin].max()) < 64 * 2.0 ** -24 * (1 + float(want[fin].abs().max()))
