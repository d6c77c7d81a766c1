"""Columns that alternate between two results."""
import pytest
import torch

from vllm_b200 import ops


@pytest.mark.parametrize("lead", [(0,), (1,), (5,), (2, 0), (2, 3)])
@pytest.mark.parametrize("n,run", [(16, 8), (24, 3), (512, 128)])
@pytest.mark.parametrize("sliced", [False, True])
def test_runs_apart(lead, n, run, sliced):
    x = torch.randn(*lead, n + 8)[..., :n] if sliced else torch.randn(*lead, n)
    a, b = ops.unzip(x, run)
    want = x.unflatten(-1, (n // (2 * run), 2, run)).movedim(-2, 0).flatten(-2)
    assert torch.equal(a, want[0]) and torch.equal(b, want[1])
