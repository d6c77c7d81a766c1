"""Requests that come to, or leave, an engine whose steps run one ahead."""
import pytest

from tests.test_run_ahead import PROMPTS, _same, _stepped
from tests.utils import make_llm
from vllm_b200 import SamplingParams

GREEDY = SamplingParams(max_tokens=12, temperature=0.0, ignore_eos=True)
JOINS = {"penalty": SamplingParams(max_tokens=9, temperature=0.0, ignore_eos=True, repetition_penalty=1.3), "plain": GREEDY,
         "bias": SamplingParams(max_tokens=9, temperature=0.0, ignore_eos=True, min_tokens=2, logit_bias={7: 3.0}),
         "prompt": SamplingParams(max_tokens=3, temperature=0.0, ignore_eos=True, prompt_logprobs=2)}


def check(llm, joins, at=3):
    core = llm.llm_engine.engine_core.engine_core
    want = _stepped(llm, PROMPTS[:5], GREEDY)
    extra = _stepped(llm, PROMPTS[5:6], joins)
    step, seen = llm.llm_engine.step, []

    def stepping():
        seen.append(core._ahead)
        if len(seen) == at:
            seen.extend(llm._add(PROMPTS[5:6], joins, None, None, final_only=True))
        return step()
    llm.llm_engine.step = stepping
    try:
        outs = llm.generate(PROMPTS[:5], GREEDY)
    finally:
        llm.llm_engine.step = step
    _same(outs[:5], want)
    _same(outs[5:], extra)
    assert (outs[5].prompt_logprobs is None) == (extra[0].prompt_logprobs is None)
    assert seen[0] and core.batch_queue is None and not core._ahead and not core.scheduler.async_scheduling and not core.scheduler.requests
    assert core.step_fn == core.step
    _same(llm.generate(PROMPTS[:5], GREEDY), want)


def check_abort(llm):
    core = llm.llm_engine.engine_core.engine_core
    want = _stepped(llm, PROMPTS[:5], GREEDY)
    step, n, gone = llm.llm_engine.step, [0], []

    def stepping():
        n[0] += 1
        if n[0] == 5:
            gone.append(sorted(llm.llm_engine.output_processor.request_states, key=int)[1])
            llm.llm_engine.abort_request(gone)
        return step()
    llm.llm_engine.step = stepping
    try:
        outs = {o.request_id: o for o in llm.generate(PROMPTS[:5], GREEDY)}
    finally:
        llm.llm_engine.step = step
    left = [str(int(gone[0]) - 1 + i) for i in (0, 2, 3, 4)]
    _same([outs[i] for i in left], [want[i] for i in (0, 2, 3, 4)])
    assert core.batch_queue is None and not core.scheduler.requests
    _same(llm.generate(PROMPTS[:5], GREEDY), want)


@pytest.mark.parametrize("joins", JOINS)
def test_a_request_joins(joins):
    check(make_llm("llama-tiny", max_num_seqs=8, max_num_batched_tokens=64), JOINS[joins])


def test_a_request_is_aborted():
    check_abort(make_llm("llama-tiny", max_num_seqs=8, max_num_batched_tokens=64))
