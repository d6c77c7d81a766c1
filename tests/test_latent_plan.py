"""Latent attention of prompts: what a step holds beside its activations stays within what the memory-profiling run held."""
import random
from types import SimpleNamespace

import pytest
import torch

from vllm_b200.layers import latent
from vllm_b200.layers.latent import LatentForms, LatentPlan, grouped


class _Layer(LatentForms):
    def __init__(self, heads, dim, rot, v_dim, kv_rank, window, apart):
        self.heads, self.dim, self.rot, self.v_dim, self.kv_rank, self.window, self.kv_apart = heads, dim, rot, v_dim, kv_rank, window, apart


def _metadata(q_lens, seq_lens):
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    return SimpleNamespace(host_lens=(cu, seq_lens), latent_plan=None, block_table=torch.arange(len(q_lens))[:, None].repeat(1, 3))


@pytest.mark.parametrize("window,apart", [(0, 128), (0, 1), (64, 1)])
@pytest.mark.parametrize("limit", [1 << 13, 1 << 17, 1 << 30])
def test_steps_stay_within_the_profiled_bytes(window, apart, limit, monkeypatch):
    monkeypatch.setattr(latent, "EXPAND_BYTES", limit)
    layer, rng = _Layer(4, 16, 8, 16, 32, window, apart), random.Random(limit + window)
    for _ in range(200):
        requests, tokens, length = rng.randint(1, 12), rng.choice([16, 40, 256, 2048]), rng.choice([20, 130, 1000, 5000])
        q_lens, left = [], tokens
        while left and len(q_lens) < requests:
            q_lens.append(min(left, length, rng.choice([1, 5, 17, 18, 100, 400])))
            left -= q_lens[-1]
        seq_lens = [rng.randint(n, length) for n in q_lens]
        plan = LatentPlan.of(_metadata(q_lens, seq_lens), torch.device("cpu"), window, apart, layer._most_rows(2))
        bound = layer.expanded_bytes(requests, tokens, length, 2)
        for c in plan.contexts:
            step = layer._heads_at_a_time(c.num_kv, 2)
            assert c.num_kv * (32 + 8) * 2 + step * c.num_kv * (16 + 16) * 2 <= bound
        # every portion above the absorbed form's length is in one group, in order, with its own rows
        long = [i for i, n in enumerate(q_lens) if n > latent.ABSORB_MAX_TOKENS]
        assert [int(r) for c in plan.contexts for r in c.block_table[:, 0]] == long
        for c in plan.contexts:
            assert c.cu_kv[0] == 0 and int(c.cu_kv[-1]) == c.num_kv and c.max_q == int(c.q_len.max())
            assert c.max_kv == int((c.cu_kv[1:] - c.cu_kv[:-1]).max()) and bool((c.cu_kv[1:] - c.cu_kv[:-1] >= c.seq_len).all())
            assert c.cu_kv.tolist()[:-1] == [n for n in c.cu_kv.tolist()[:-1] if n % apart == 0]
        firsts = [int(x) for c in plan.contexts for x in (c.kv_first if c.kv_first is not None else torch.zeros_like(c.q_len))]
        assert firsts == [max(seq_lens[i] - q_lens[i] + 1 - window, 0) if window else 0 for i in long]
        assert [int(x) for c in plan.contexts for x in c.seq_len] == [seq_lens[i] - f for i, f in zip(long, firsts)]
        assert plan.num_rows == sum(n for n in q_lens if n <= latent.ABSORB_MAX_TOKENS)


def test_groups():
    assert grouped([], 5) == [] and grouped([9], 5) == [(0, 1)]
    assert grouped([2, 3, 1, 9, 1, 4], 5) == [(0, 2), (2, 3), (3, 4), (4, 6)]


@pytest.mark.gpu
def test_groups_of_contexts_change_nothing(monkeypatch):
    from tests.test_e2e_gpu import PROMPTS, _llm
    from vllm_b200 import SamplingParams
    sp = SamplingParams(max_tokens=4, temperature=0.0, ignore_eos=True, prompt_logprobs=0)
    llm, runner = _llm("deepseek-small", enforce_eager=True)
    got = []
    for limit in (1 << 30, 1 << 17):                # all heads and requests at once; a request and a head at a time
        monkeypatch.setattr(latent, "EXPAND_BYTES", limit)
        outs = llm.generate(PROMPTS, sp)
        got.append([lp[t].logprob for o in outs for lp, t in zip(o.prompt_logprobs[1:], o.prompt_token_ids[1:])])
    llm.shutdown()
    # (products of other sizes round otherwise, and an expert's choice may turn on that)
    diffs = sorted(abs(a - b) for a, b in zip(*got))
    assert diffs[len(diffs) // 2] < 0.01 and diffs[int(0.9 * len(diffs))] < 0.1, diffs[-5:]


@pytest.mark.gpu
def test_long_contexts_in_small_portions_stay_within_the_profile():
    """Portions of 256 tokens over contexts of 3500."""
    from tests.test_e2e_gpu import _llm
    from vllm_b200 import SamplingParams
    llm, runner = _llm("deepseek-small", enforce_eager=True, max_model_len=4096, max_num_batched_tokens=256)
    dev = runner.device
    sp = SamplingParams(max_tokens=1, temperature=0.0, ignore_eos=True)
    base = torch.cuda.memory_allocated(dev)
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats(dev)
    runner.profile_run()
    profiled = torch.cuda.max_memory_allocated(dev) - base
    torch.cuda.reset_peak_memory_stats(dev)
    llm.generate([{"prompt_token_ids": [(13 * i + j) % 4000 + 5 for j in range(3500)]} for i in range(6)], sp)
    assert torch.cuda.max_memory_allocated(dev) - base <= profiled
    llm.shutdown()
