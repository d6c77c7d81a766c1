"""Run-ahead beside synchronous steps for models with windows, latents, experts and recurrent states: more requests than run together, requests that lose
their pages on the way, requests that join, one that is aborted.  Weights as in ``perf/cases.py``: the likeliest token stands clear of the second."""
import pytest

from tests.test_run_ahead import _stepped
from vllm_b200 import SamplingParams

pytestmark = pytest.mark.gpu
PROMPTS = [{"prompt_token_ids": [(131 * i + 7 * j) % 30000 + 5 for j in range(15 + 41 * i)]} for i in range(7)]


def _llm(family, blocks):
    from perf import cases
    from vllm_b200 import LLM
    c = {"family": family, "width": 1024, "fp8": False}
    return LLM(cases._checkpoint(c), dtype="bfloat16", skip_tokenizer_init=True, max_model_len=512, max_num_seqs=4, max_num_batched_tokens=160,
               kv_cache_memory_bytes=1 << 30, cudagraph_capture_sizes=[1, 2, 4], multiprocess_mode=False, enable_prefix_caching=False,
               **({} if blocks is None else {"num_gpu_blocks_override": blocks}))


def _same(got, want):
    """Steps have other companions than synchronous ones, so that 16 bits round differently: half a unit of a logit of up to 16."""
    for x, y in zip(got, want, strict=True):
        x, y = x.outputs[0], y.outputs[0]
        assert x.token_ids == y.token_ids and x.finish_reason == y.finish_reason and x.stop_reason == y.stop_reason
        for p, q in zip(x.logprobs or [], y.logprobs or [], strict=True):
            t = max(q, key=lambda i: q[i].logprob)
            assert abs(p[t].logprob - q[t].logprob) < 2.0 ** -5 * 2


@pytest.mark.parametrize("family,blocks", [("gemma2", None), ("gemma2", 26), ("mixtral", 14), ("deepseek", None), ("deepseek", 14), ("qwen3next", None), ("qwen3next", 14)])
def test_same_as_synchronous_steps(family, blocks):
    llm = _llm(family, blocks)
    eng, core = llm.llm_engine, llm.llm_engine.engine_core.engine_core
    greedy = SamplingParams(max_tokens=60, temperature=0.0, ignore_eos=True, logprobs=2)
    want = _stepped(llm, PROMPTS, greedy)
    before = core.scheduler._num_preemptions
    _same(llm.generate(PROMPTS, greedy), want)
    assert (blocks is None) == (core.scheduler._num_preemptions == before)
    # ended by a token at different steps
    params = [SamplingParams(max_tokens=20, temperature=0.0, ignore_eos=True, stop_token_ids=[w.outputs[0].token_ids[3 + 2 * i]]) for i, w in enumerate(want)]
    _same(llm.generate(PROMPTS, params), _stepped(llm, PROMPTS, params))
    # one leaves, one joins that ends the run-ahead
    biased = SamplingParams(max_tokens=9, temperature=0.0, ignore_eos=True, logit_bias={7: 1.0})
    late = _stepped(llm, PROMPTS[2:3], biased)
    step, seen = eng.step, []

    def stepping():
        seen.append(core._ahead)
        if len(seen) == 6:
            eng.abort_request([sorted(eng.output_processor.request_states, key=int)[0]])
        if len(seen) == 12:
            llm._add(PROMPTS[2:3], biased, None, None, final_only=True)
        return step()
    eng.step = stepping
    try:
        outs = [o for o in llm.generate(PROMPTS, greedy) if o.outputs[0].finish_reason != "abort"]
    finally:
        eng.step = step
    assert seen[0] and not seen[-1]
    _same(outs, want[1:] + late)
    assert core.batch_queue is None and not core.scheduler.requests
    llm.shutdown()
