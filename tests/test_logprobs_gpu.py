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
