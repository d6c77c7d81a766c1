"""VLLM_BATCH_INVARIANT=1: a row's log-probabilities and its experts do not depend on the rows beside it, nor on how many likeliest tokens others ask for."""
import pytest
import torch

from tests.test_batch_invariant_gpu import _mode  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1000, 32000, 128256, 262145])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_log_probabilities(V, dtype):
    from vllm_b200.ops import cuda as cu
    n = 7_500_000 // V + 2                           # rows beyond which the default dispatch takes another form
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(min(n, 300), V, device="cuda", generator=g).mul_(3).to(dtype)
    picked = torch.randint(0, V, (len(x),), device="cuda", generator=g)
    first = min(len(x), 64)
    alone = torch.cat([cu.logprobs(x[i:i + 1], picked[i:i + 1], 5) for i in range(first)])
    for rows in {min(first, 2), first, len(x) - 2, len(x)}:
        for k in (0, 1, 8, 9, 64 if V < 40000 else 11):
            got, want, m = cu.logprobs(x[:rows], picked[:rows], k)[:first], alone[:rows], min(k, 5)
            assert torch.equal(got[:, :m + 1], want[:, :m + 1])                                     # places
            assert torch.equal(got[:, k + 1:k + 2 + m], want[:, 6:7 + m])                           # bits of the numbers
            assert torch.equal(got[:, -1], want[:, -1])


@pytest.mark.parametrize("E,groups,keep", [(160, 8, 3), (256, 1, 1), (64, 4, 2)])
@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_experts_of_a_token(E, groups, keep, scoring):
    from vllm_b200.ops import cuda as cu
    lg = torch.randn(1500, E, device="cuda", generator=torch.Generator(device="cuda").manual_seed(E)) * 3
    few, many = (cu.grouped_topk(lg[:n], 6, groups, keep, True, scoring, None, 1.0) for n in (8, 1500))
    assert torch.equal(few[0], many[0][:8]) and torch.equal(few[1], many[1][:8])
