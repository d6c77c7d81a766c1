"""VLLM_BATCH_INVARIANT=1: bits of the same rows alone and inside batches above every threshold of the default dispatch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _mode(monkeypatch):
    from vllm_b200 import envs
    from vllm_b200.ops import cuda as cu
    monkeypatch.setenv("VLLM_BATCH_INVARIANT", "1")
    envs._cache.clear()
    envs.disable_envs_cache()
    cu._plan_cache.clear()
    cu._fp8_plan_cache.clear()
    yield
    envs._cache.clear()
    cu._plan_cache.clear()
    cu._fp8_plan_cache.clear()


def _rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("H", [1024, 2048, 4096, 8192])
@pytest.mark.parametrize("gemma", [False, True])
def test_norms(H, gemma):
    from vllm_b200.ops import cuda as cu
    big, n, k = 1300, 300, 3                                       # more threads per row than rows leave, below and above 1024 rows
    x, r, y = _rnd(big, H), _rnd(big, H, seed=1), _rnd(big * k, H, seed=2)
    w, v = _rnd(H, seed=3), _rnd(H, seed=4)
    inv = torch.arange(big * k, dtype=torch.int32, device="cuda")
    tw = torch.rand(big, k, device="cuda")
    runs = {"norm": lambda m: (cu.rms_norm(x[:m], w, 1e-6, gemma),),
            "add": lambda m: cu.fused_add_rms_norm(x[:m].clone(), r[:m].clone(), w, 1e-6, gemma),
            "tail": lambda m: cu.norm_add_norm(x[:m], r[:m].clone(), w, 1e-6, v, 1e-5, gemma),
            "experts": lambda m: cu.moe_combine_norm(y[:m * k], inv[:m * k], tw[:m], r[:m].clone(), w, 1e-6, gemma, x[:m])}
    for name, run in runs.items():
        for a, b in zip(run(n), run(big)):
            assert torch.equal(a, b[:n]), name
