"""Stored pages of models whose page layout changed are not found under the names of the old layout; other models' names stay."""
import hashlib
import json
from types import SimpleNamespace as NS

import pytest

from vllm_b200.kv_transfer import BlockConnector


def _old(model, hf, size):
    ident = {"model": model, "dtype": "torch.bfloat16", "kv_dtype": "auto", "block_size": size, "tp": 1, "pp": 1, "dcp": 1, "hf": hf}
    return hashlib.sha256(json.dumps(ident, sort_keys=True, default=str).encode()).hexdigest()[:12]


@pytest.mark.parametrize("hf,size,kept", [({"hidden_size": 64}, 64, True), ({"attn_logit_softcapping": None}, 64, True),
                                          ({"final_logit_softcapping": 30.0}, 64, True), ({"attn_logit_softcapping": 50.0}, 32, True),
                                          ({"attn_logit_softcapping": 50.0}, 64, False),
                                          ({"text_config": {"attn_logit_softcapping": 50.0}}, 64, False)])
def test_names_follow_the_layout(hf, size, kept):
    cfg = NS(kv_transfer_config=NS(kv_role=None), cache_config=NS(block_size=size, cache_dtype="auto"),
             model_config=NS(model="m", torch_dtype="torch.bfloat16", hf_config=hf),
             parallel_config=NS(tensor_parallel_size=1, pipeline_parallel_size=1, decode_context_parallel_size=1))
    assert (BlockConnector(cfg, "scheduler", None)._ns == _old("m", hf, size)) is kept
