"""Several layers of one input: together where nothing forbids it."""
import pytest
import torch

from tests.utils import make_llm
from vllm_b200 import SamplingParams, ops
from vllm_b200.layers.linear import ReplicatedLinear, products


def test_hooks_of_a_layer_are_called(monkeypatch):
    a, b = (ReplicatedLinear(16, n, dtype=torch.float32) for n in (8, 4))
    x = torch.randn(3, 16)
    with torch.no_grad():
        for m in (a, b):
            m.weight.normal_()
    together = []
    monkeypatch.setattr(ops, "linear_parts", lambda x, ws, bs, forms: together.append(1) or [x @ w.t() for w in ws])
    want = [x @ m.weight.t() for m in (a, b)]
    assert all(torch.equal(p, q) for p, q in zip(products(x, (a, None), (b, None)), want)) and together == [1]
    for put in (b.register_forward_hook, lambda f: b.register_forward_pre_hook(lambda m, args: f(m, args, None))):
        seen = []
        hook = put(lambda m, args, out: seen.append(m) or None)
        got = products(x, (a, None), (b, None))
        assert seen == [b] and together == [1] and all(torch.allclose(p, q) for p, q in zip(got, want))
        hook.remove()
    products(x, (a, None), (b, None))
    assert together == [1, 1]


@pytest.mark.parametrize("preset,name", [("deepseek-tiny", "shared_experts"), ("qwen2moe-tiny", "shared_expert")])
def test_hooks_of_shared_experts_are_called(preset, name):
    llm = make_llm(preset)
    model = llm.llm_engine.engine_core.engine_core.model_executor.worker.runner.model
    prompt, sp = [{"prompt_token_ids": list(range(5, 25))}], SamplingParams(max_tokens=3, temperature=0.0, ignore_eos=True)
    want = llm.generate(prompt, sp)[0].outputs[0].token_ids
    blocks = [m for n, m in model.named_modules() if n.endswith("." + name)]
    seen = []
    hooks = [m.register_forward_hook(lambda m, args, out: seen.append(m) or None) for m in blocks]
    assert llm.generate(prompt, sp)[0].outputs[0].token_ids == want
    assert blocks and set(seen) == set(blocks)
    for h in hooks:
        h.remove()
