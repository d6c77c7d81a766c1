"""How many key ranges a decode step has: what is asked for is what runs."""
import pytest

from vllm_b200 import envs
from vllm_b200.ops import cuda as cu


@pytest.mark.parametrize("asked", [3, 5, 16])
def test_forced_splits_are_not_cut(asked, monkeypatch):
    monkeypatch.setenv("VLLM_B200_ATTN_SPLITS", str(asked))
    assert envs.VLLM_B200_ATTN_SPLITS == asked
    assert cu.decode_splits(2, 8, 1 << 17, 128) == asked and cu.mla_decode_splits(2, 128, 1 << 15) == asked
