"""Log-probabilities of generated tokens are those that were recorded: kernels for the same step may be exchanged, its roundings stay.

``tests/data/logprobs.json`` holds, per case, the five likeliest tokens' log-probabilities of every request's last generated token, from the tree of before the decode
kernels with warp-level products, which changed the third digit of most of them.  Weights and prompts are those of ``perf/cases.py``."""
import json
import os

import pytest
import torch

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(__file__)
CASES = {"llama": ("llama", 12, 20, 90, 5, False), "llama long": ("llama", 3, 500, 700, 3, False), "llama fp8": ("llama", 12, 20, 90, 5, True),
         "gemma2": ("gemma2", 12, 20, 90, 5, False), "gemma2 long": ("gemma2", 3, 500, 700, 3, False), "mixtral": ("mixtral", 12, 20, 90, 5, False),
         "deepseek": ("deepseek", 12, 20, 90, 5, False), "deepseek long": ("deepseek", 3, 500, 700, 3, False), "qwen3next": ("qwen3next", 12, 20, 90, 5, False)}


def outputs(name):
    from perf import cases
    family, requests, low, high, new, fp8 = CASES[name]
    state = cases.prepare({"family": family, "width": 1024, "requests": requests, "low": low, "high": high, "new": new, "logprobs": True, "fp8": fp8}, 3)
    return cases.run(state)["logprobs"][:, -1]


@pytest.mark.parametrize("name", CASES)
def test_outputs_are_the_recorded_ones(name):
    with open(os.path.join(HERE, "data", "logprobs.json")) as f:
        data = json.load(f)
    if data["torch"] != torch.__version__:
        pytest.skip("weights and prompts come from another generator")
    want, got = torch.tensor(data[name], dtype=torch.float64), outputs(name).double()
    # steps repeat exactly but for the sums of the log-probabilities themselves, in 32 bits and any order
    assert float((got - want).norm() / want.norm()) < 2e-5
