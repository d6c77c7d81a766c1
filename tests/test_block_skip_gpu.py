"""Streams that a model keeps for a later layer (Solar's block skips) beside fused kernels that add to the stream in place."""
import pytest

from tests.test_e2e_gpu import PROMPTS, _llm

pytestmark = pytest.mark.gpu


def test_block_skips_match_the_reference_ops(monkeypatch):
    from vllm_b200 import SamplingParams
    sp = SamplingParams(max_tokens=1, temperature=0.0, ignore_eos=True, prompt_logprobs=0)

    def logprobs(tv, ref=False):
        monkeypatch.setenv("VLLM_B200_FORCE_REF_OPS", str(int(ref)))
        llm, _ = _llm(enforce_eager=True, hf_overrides=dict(architectures=["SolarForCausalLM"], bskcn_1=[1], bskcn_2=[0], bskcn_3=[3], bskcn_4=[2],
                                                            bskcn_tv=[0.9, tv]))
        outs = llm.generate(PROMPTS, sp)
        llm.shutdown()
        return [lp[t].logprob for o in outs for lp, t in zip(o.prompt_logprobs[1:], o.prompt_token_ids[1:])]
    got, want, plain = logprobs(0.7), logprobs(0.7, ref=True), logprobs(0.0)
    far = lambda a, b: sum(abs(x - y) for x, y in zip(a, b)) / len(a)  # noqa: E731
    # the skips change the result; with them the two implementations differ by the rounding of 16-bit activations only
    assert far(want, plain) > 10 * far(got, want), (far(got, want), far(want, plain))
