"""A kernel that gave up on a wait ends the step with an error instead of tokens."""
import numpy as np
import pytest

from tests.utils import make_llm
from vllm_b200 import SamplingParams


def _runner(llm):
    return llm.llm_engine.engine_core.engine_core.model_executor.worker.runner


@pytest.mark.parametrize("when", ["launch", "result"])
def test_step_raises(when, monkeypatch):
    llm = make_llm("llama-tiny", max_num_seqs=4)
    runner = _runner(llm)
    assert runner.kernel_error is None               # (no device, no flag)
    runner.kernel_error = np.zeros(1, dtype=np.int32)
    sp, prompt = SamplingParams(max_tokens=3, temperature=0.0, ignore_eos=True), [{"prompt_token_ids": [5, 9, 30]}]
    want = llm.generate(prompt, sp)[0].outputs[0].token_ids
    if when == "launch":                             # by a step whose results this rank does not read
        runner.kernel_error[0] = 1
    else:
        forward = runner._forward

        def gives_up(*a, **kw):
            out = forward(*a, **kw)
            runner.kernel_error[0] = 1
            return out
        monkeypatch.setattr(runner, "_forward", gives_up)
    with pytest.raises(RuntimeError, match="gave up"):
        llm.generate(prompt, sp)
    assert runner.kernel_error[0] == 0
    llm.shutdown()


@pytest.mark.gpu
@pytest.mark.parametrize("eager", [True, False])
def test_flag_is_there_before_the_first_capture(eager):
    import torch
    from tests.test_e2e_gpu import PROMPTS, _llm
    from vllm_b200.ops import cuda_ops
    llm, runner = _llm(enforce_eager=eager, cudagraph_capture_sizes=[8])
    flag = cuda_ops().kernel_error_flag(torch.device("cuda", 0))
    assert flag.is_pinned() and flag.numpy().ctypes.data == runner.kernel_error.ctypes.data
    sp = SamplingParams(max_tokens=4, temperature=0.0, ignore_eos=True)
    assert len(llm.generate(PROMPTS, sp)[0].outputs[0].token_ids) == 4
    runner.kernel_error[0] = 1
    with pytest.raises(RuntimeError, match="gave up"):
        llm.generate(PROMPTS, sp)
    llm.shutdown()


@pytest.mark.gpu
def test_kernels_store_into_pinned_memory():
    """Where the flag lies: a kernel's store is there behind the event that follows it."""
    import torch
    from vllm_b200.ops import cuda as cu
    x, out = torch.zeros(1, 64, device="cuda"), torch.zeros(3, dtype=torch.int32, pin_memory=True)
    x[0, 7] = 3.0
    sampled = torch.tensor([7], device="cuda")
    cu._check(cu._logprobs(x.data_ptr(), 64, 1, 64, sampled.data_ptr(), 0, out.data_ptr(), cu._DT[x.dtype], cu._st()), "logprobs")
    done = torch.cuda.Event()
    done.record()
    done.synchronize()
    assert out[0] == 7 and out[2] == 1
