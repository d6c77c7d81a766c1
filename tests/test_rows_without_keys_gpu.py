"""Decode attention of rows that have no keys (yet): zeros, and a log-sum-exp of nothing or of the sink."""
import pytest
import torch

from tests.test_kernels_gpu import _mk_attn_case, _to_tc_layout, cu

pytestmark = pytest.mark.gpu


def _stale(*shapes, dtype):
    """Memory that an allocation without values finds next holds NaN."""
    for t in [torch.full(s, float("nan"), device="cuda", dtype=dtype) for s in shapes]:
        del t


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("Hq,Hkv", [(8, 8), (8, 2), (32, 2)])
def test_rows(dtype, splits, sink, Hq, Hkv):
    lens = [1, 70, 300, 5]
    q, cache, md = _mk_attn_case(4, Hq, Hkv, 128, 64, lens, [1] * 4, dtype=dtype)
    md.kv_vt, md.num_splits, md.max_seq_len = True, splits, 300
    sinks = torch.randn(Hq, device="cuda") if sink else None
    full, full_lse = cu().paged_attention(q, _to_tc_layout(cache), md, 0.09, sinks=sinks, return_lse=True)
    md.seq_lens = md.seq_lens.clone()
    md.seq_lens[[0, 2]] = 0
    tc = _to_tc_layout(cache)
    _stale(full.shape, dtype=dtype)
    _stale(full_lse.shape, dtype=torch.float32)
    got, lse = cu().paged_attention(q, tc, md, 0.09, sinks=sinks, return_lse=True)
    assert bool((got[[0, 2]] == 0).all()) and torch.equal(got[[1, 3]], full[[1, 3]]) and torch.equal(lse[[1, 3]], full_lse[[1, 3]])
    if sink:
        assert torch.allclose(lse[[0, 2]], sinks.expand(2, Hq), rtol=1e-6, atol=1e-6)
    else:
        assert bool((lse[[0, 2]] == float("-inf")).all())


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("R,P,H", [(512, 64, 16), (72, 40, 17), (512, 0, 128)])
def test_rows_of_latents(splits, R, P, H):
    lens = torch.tensor([1, 70, 300, 5], dtype=torch.int32, device="cuda")
    q, qp = torch.randn(4, H, R, device="cuda").bfloat16(), torch.randn(4, H, P, device="cuda").bfloat16() if P else None
    cache, bt = torch.randn(25, 64, R + P, device="cuda").bfloat16(), torch.arange(1, 25, dtype=torch.int32, device="cuda").view(4, 6)
    run = lambda n: cu().mla_decode_tc(q, qp, cache, bt, n, 0.05, 300, splits, return_lse=True)          # noqa: E731
    full, full_lse = run(lens)
    lens = lens.clone()
    lens[[0, 2]] = 0
    _stale(full.shape, dtype=full.dtype)
    _stale(full_lse.shape, dtype=torch.float32)
    got, lse = run(lens)
    assert bool((got[[0, 2]] == 0).all()) and bool((lse[[0, 2]] == float("-inf")).all())
    assert torch.equal(got[[1, 3]], full[[1, 3]]) and torch.equal(lse[[1, 3]], full_lse[[1, 3]])
