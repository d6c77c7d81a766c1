"""``generate`` launches a step while the one before is on the device; its results are those of synchronous steps."""
import copy

import pytest

from tests.utils import make_llm
from vllm_b200 import SamplingParams


def _stepped(llm, prompts, params):
    """The same requests through the engine's own synchronous steps."""
    ids = llm._add(prompts, params, None, None, final_only=True)
    outs = {}
    while llm.llm_engine.has_unfinished_requests():
        for o in llm.llm_engine.step():
            outs[o.request_id] = o
    return [outs[i] for i in ids]


def _same(a, b):
    for x, y in zip(a, b, strict=True):
        x, y = x.outputs[0], y.outputs[0]
        assert x.token_ids == y.token_ids and x.finish_reason == y.finish_reason and x.stop_reason == y.stop_reason
        assert (x.logprobs is None) == (y.logprobs is None)
        for p, q in zip(x.logprobs or [], y.logprobs or []):
            assert p.keys() == q.keys() and all(abs(p[t].logprob - q[t].logprob) < 1e-3 for t in p)


PROMPTS = [{"prompt_token_ids": [(13 * i + 7 * j) % 90 + 5 for j in range(5 + 9 * i)]} for i in range(7)]


def _check(llm):
    core = llm.llm_engine.engine_core.engine_core
    greedy = SamplingParams(max_tokens=12, temperature=0.0, ignore_eos=True)
    base = _stepped(llm, PROMPTS, greedy)
    seen = []
    run, core.step_with_batch_queue = core.step_with_batch_queue, lambda: (seen.append(len(core.batch_queue)), run())[1]
    _same(llm.generate(PROMPTS, greedy), base)
    assert seen
    assert core.batch_queue is None and not core.scheduler.async_scheduling and not core.scheduler.requests
    # requests of all kinds beside each other: ended by a token after different steps, seeded, with log-probabilities
    stop = [o.outputs[0].token_ids[2 + i % 4] for i, o in enumerate(base)]
    params = [SamplingParams(max_tokens=3 + i, temperature=0.0 if i % 2 else 0.9, seed=i, ignore_eos=True, stop_token_ids=[stop[i]],
                             logprobs=2 if i % 3 == 0 else None) for i in range(len(PROMPTS))]
    _same(llm.generate(PROMPTS, params), _stepped(llm, PROMPTS, params))
    # host state per token: synchronous steps
    seen.clear()
    held = [SamplingParams(max_tokens=6, temperature=0.0, ignore_eos=True, repetition_penalty=1.3)] * len(PROMPTS)
    _same(llm.generate(PROMPTS, held), _stepped(llm, PROMPTS, held))
    assert not seen
    # an error leaves the engine usable
    execute = core.model_executor.execute_model
    calls = iter(range(100))

    def fails(so, non_block=False):
        if next(calls) == 3:
            raise ValueError("planted")
        return execute(so, non_block=non_block)
    core.model_executor.execute_model = fails
    with pytest.raises(ValueError, match="planted"):
        llm.generate(PROMPTS, greedy)
    core.model_executor.execute_model = execute
    assert core.batch_queue is None and not core.scheduler.requests and not llm.llm_engine.has_unfinished_requests()
    _same(llm.generate(PROMPTS, greedy), base)


def test_same_as_synchronous_steps():
    _check(make_llm("llama-tiny", max_num_seqs=4, max_num_batched_tokens=64))          # (admissions and portions of prompts in between)


def test_clones_share_nothing():
    sp = SamplingParams(n=2, stop=["a"], stop_token_ids=[3], logit_bias={1: 2.0}, allowed_token_ids=[1], bad_words=["x"], extra_args={"k": [1]})
    sp.bad_words_token_ids, sp.note = [[1, 2]], {"v": [4]}
    was, c = copy.deepcopy(sp), sp.clone()
    assert c == sp and vars(c) == vars(was) and sp.note == {"v": [4]}
    for name in ("stop", "stop_token_ids", "allowed_token_ids", "bad_words", "all_stop_token_ids"):
        getattr(c, name).append(9)
    c.bad_words_token_ids[0].append(9)
    c.logit_bias[5] = 1.0
    c.extra_args["k"].append(9)
    assert sp == was


@pytest.mark.parametrize("caching", [False, True])
@pytest.mark.parametrize("kinds", ["full,window", "window", "full,state", "full,window,state"])
def test_pages_of_several_groups(kinds, caching):
    """What neither takes a page nor gives one back is told without going through the groups' lists; the pages are those of the long way."""
    import random
    from vllm_b200.core.kv_cache_manager import FullAttentionSpec, KVCacheConfig, KVCacheGroupSpec, KVCacheManager, MambaSpec, SlidingWindowSpec
    from vllm_b200.core.request import Request
    if "state" in kinds and caching:
        pytest.skip("states are not cached by prefix")
    make = {"full": lambda: FullAttentionSpec(16, 1, 64, 2), "window": lambda: SlidingWindowSpec(16, 1, 64, 2, sliding_window=40),
            "state": lambda: MambaSpec(16, 1024)}
    both = []
    for long_way in (False, True):
        cfg = KVCacheConfig(num_blocks=60, num_state_slots=9 if "state" in kinds else 0, kv_cache_tensors=[],
                            kv_cache_groups=[KVCacheGroupSpec([k], make[k](), {}) for k in kinds.split(",")])
        kv = KVCacheManager(cfg, 400, enable_caching=caching)
        if long_way:
            for m in kv.managers:
                m.settled = lambda *a: False
        rng, live, seen, n = random.Random(3), [], [], 0
        for _ in range(600):
            if len(live) < 6 and rng.random() < 0.2:
                n += 1
                r = Request(str(n), [rng.randint(0, 3) for _ in range(rng.randint(1, 90))],
                            SamplingParams(max_tokens=200), block_hasher=kv.block_hasher)
                done, hit = kv.get_computed_blocks(r) if caching else (kv.empty_blocks(), 0)
                got = kv.allocate_slots(r, r.num_tokens - hit, hit, done)
                seen.append(None if got is None else kv.get_block_ids(r.request_id))
                if got is not None:
                    r.num_computed_tokens = r.num_tokens
                    live.append(r)
            for r in list(live):
                r.append_output_token_ids(rng.randint(0, 3))
                got = kv.allocate_slots(r, 1)
                seen.append((r.request_id, None if got is None else kv.get_block_ids(r.request_id), kv.pool.get_num_free_blocks()))
                if got is None or rng.random() < 0.01 or r.num_tokens > 380:
                    kv.free(r)
                    live.remove(r)
                else:
                    r.num_computed_tokens += 1
        both.append(seen)
    assert both[0] == both[1]


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [None, 24])          # 24: some requests lose their pages on the way and are computed again
def test_same_on_the_device(blocks):
    from tests.test_e2e_gpu import _llm
    kw = {} if blocks is None else dict(num_gpu_blocks_override=blocks)
    llm, _ = _llm(max_num_seqs=4, max_num_batched_tokens=128, max_model_len=256, cudagraph_capture_sizes=[1, 2, 4], **kw)
    _check(llm)
    llm.shutdown()
