"""Passes over a prompt's rows: sort by expert, rows to their experts, runs apart."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,k,E", [(4097, 1, 3), (4098, 6, 32), (41400, 6, 32), (8192, 8, 4096), (70000, 7, 1000), (65544, 2, 1)])
@pytest.mark.parametrize("mapped", [False, True])
def test_pairs_sorted_by_expert(R, k, E, mapped):
    from vllm_b200.ops import cuda as cu
    R = R // k * k
    g = torch.Generator(device="cuda").manual_seed(R + E)
    ids = torch.randint(0, E, (R // k, k), device="cuda", generator=g, dtype=torch.int32)
    emap = None
    if mapped:                                   # every third expert is another rank's
        emap = torch.where(torch.arange(E, device="cuda") % 3 == 2, -1, torch.arange(E, device="cuda")).int()
    tok, inv, offs, pairs = cu.moe_align(ids, E, emap, with_pairs=True)
    flat = ids.reshape(-1).long() if emap is None else emap[ids.reshape(-1).long()].long()
    n = torch.bincount(flat[flat >= 0], minlength=E)
    assert torch.equal(offs.long(), torch.cat([n.new_zeros(1), n.cumsum(0)]))
    here = (flat >= 0).nonzero().flatten()
    p = inv.long()
    assert bool((p[flat < 0] == -1).all()) and torch.equal(p[here].sort().values, torch.arange(len(here), device="cuda"))
    assert bool(((offs[flat[here]] <= p[here]) & (p[here] < offs[flat[here] + 1])).all())
    assert torch.equal(pairs.long()[p[here]], here) and torch.equal(tok.long()[p[here]], here // k)
    assert bool((tok[len(here):] == 0).all()) and bool((pairs[len(here):] == 0).all())


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (700, 6, 2048), (33, 2, 2056), (5, 8, 64)])
def test_rows_to_their_experts(T, k, H):
    from vllm_b200.ops import cuda as cu
    x = torch.randn(T, H, device="cuda").bfloat16()
    inv = torch.randperm(T * k, device="cuda").int()
    inv[::5] = -1
    xs = cu.moe_spread(x, inv)
    here = (inv >= 0).nonzero().flatten()
    assert torch.equal(xs[inv[here].long()], x[here // k])


@pytest.mark.parametrize("shape,run", [((1, 16), 8), ((300, 4096), 128), ((2, 3, 96), 24)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_runs_apart(shape, run, dtype):
    from vllm_b200 import ops
    x = torch.randn(shape, device="cuda").to(dtype)
    want = x.view(*shape[:-1], -1, 2, run)
    for i, y in enumerate(ops.unzip(x, run)):
        assert torch.equal(y, want[..., i, :].reshape(*shape[:-1], -1))
    odd = torch.randn(3, 12, device="cuda").to(dtype)
    assert torch.equal(ops.unzip(odd, 3)[1], odd.view(3, 2, 2, 3)[:, :, 1].reshape(3, 6))
