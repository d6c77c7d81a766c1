"""The likeliest tokens of rows whose values are equal, or lie in order: beyond what the lists of the log-probability kernel hold."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,k", [(33, 33), (2048, 64), (32000, 5), (65537, 20), (128256, 1), (131073, 64), (262144, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_equal_and_ordered_rows(V, k, dtype):
    from vllm_b200.ops import cuda as cu
    up = torch.arange(V, device="cuda").float() / V
    rows = [torch.zeros(V), torch.full((V,), -7.0), up * 8, -up * 8, torch.where(up > 0.5, 1.0, up * 0), torch.where(up < 0.3, 1.0, 0.0), up.floor(),
            torch.where(up >= 1 - 600 / V, 1 + up, 1.0), torch.full((V,), float("-inf"))]
    x = torch.stack([r.cuda().to(dtype) for r in rows])
    x[6, V - 1], x[8, V // 3] = 3.0, 2.0
    sampled = torch.arange(len(rows), device="cuda") * (V // 10)
    p = cu.logprobs(x, sampled, k)
    order = x.float().sort(dim=-1, descending=True, stable=True)
    assert torch.equal(p[:, 1:k + 1].long(), order.indices[:, :k])
    want = x.double().log_softmax(-1).gather(1, order.indices[:, :k])
    got = p[:, k + 2:2 * k + 2].contiguous().view(torch.float32).double()
    fin = want.isfinite()
    assert torch.equal(got.isfinite(), fin)
    # 32 additions in a thread, at most 13 one after the other beyond them, each 2^-24 of the sum; expf and logf a few more
    assert float((got - want).abs()[fin].max()) < 64 * 2.0 ** -24 * (1 + float(want[fin].abs().max()))


@pytest.mark.parametrize("V,k", [(33, 1), (2048, 5), (32000, 1), (32000, 64), (128256, 5), (262144, 17)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_cluster_and_a_block_choose_alike(V, k, dtype, monkeypatch):
    """Rows with NaN and infinities, too: the same places in the same order, the same ranks."""
    from vllm_b200.ops import cuda as cu
    x = torch.randn(8, V, device="cuda", generator=torch.Generator(device="cuda").manual_seed(V + k))
    x[1, ::3], x[2, :V - 20], x[3], x[4, V // 2], x[5, :V - 3] = float("nan"), float("nan"), float("nan"), float("inf"), float("-inf")
    x[6, :32] = float("nan")
    x = x.to(dtype)
    sampled = torch.full((8,), V - 1, device="cuda")
    both = [cu.logprobs(x, sampled, k)]
    monkeypatch.setattr(cu, "batch_invariant", lambda: True)
    both.append(cu.logprobs(x, sampled, k))
    a, b = both
    assert torch.equal(a[:, :k + 1], b[:, :k + 1]) and torch.equal(a[[0, 4, 5], -1], b[[0, 4, 5], -1])
    va, vb = (t[:, k + 1:-1].contiguous().view(torch.float32) for t in both)
    assert torch.equal(va.isnan(), vb.isnan()) and torch.equal(va.isinf(), vb.isinf())
    fin = va.isfinite()
    assert float((va - vb)[fin].abs().max()) < 1e-5
