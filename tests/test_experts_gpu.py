"""Grouped products of decode steps whose weights one block per SM streams."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(R, N, K, E, dtype, skew, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(R, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(E, N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    ids = torch.randint(0, E, (R,), device="cuda", generator=g)
    if skew:                                         # most experts without rows, one with many
        ids = torch.where(torch.rand(R, device="cuda", generator=g) < 0.8, E - 1, ids)
    ids = ids.sort().values
    offs = torch.searchsorted(ids, torch.arange(E + 1, device="cuda")).int()
    exact = torch.einsum("rk,rnk->rn", x.double(), w.double()[ids]) if R * N * K < 1 << 27 else torch.stack([w[e].double() @ v.double() for v, e in zip(x, ids)])
    size = torch.stack([w[e].double().abs() @ v.double().abs() for v, e in zip(x, ids)])
    return x, w, ids, offs, exact, K * 2.0 ** -24 * size       # bound of 32-bit sums in any order


@pytest.mark.parametrize("R,N,K,E,bn", [(1, 128, 64, 1, 16), (7, 128, 192, 300, 16), (40, 256, 704, 3, 16), (144, 1536, 512, 32, 16), (33, 384, 128, 512, 16), (65, 640, 1024, 2, 32),
                                        (100, 128, 640, 32, 16), (129, 256, 2048, 2, 64), (300, 256, 64, 2, 128)])
@pytest.mark.parametrize("act", [None, "silu", "gelu_tanh"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("skew", [False, True])
def test_experts(R, N, K, E, bn, act, dtype, skew):
    from vllm_b200.ops import cuda as cu
    x, w, ids, offs, exact, bound = _case(R, N, K, E, dtype, skew, R)
    y = cu.gemm_experts(x, w, offs, bn, act)
    u, tiny = (2.0 ** -8, 0.0) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    want = exact
    if act:
        gate, up = exact.chunk(2, 1)
        bg, bu = bound.chunk(2, 1)
        a = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
        want = a * up
        # slopes of at most 1.13; quick exponentials and divisions a few 2^-21 of the gate (the tanh of a sum near its end loses as much of the gate)
        bound = (1.13 * bg + 2.0 ** -19 * gate.abs()) * (up.abs() + bu) + a.abs() * bu
    assert y.shape == want.shape
    assert bool(((y.double() - want).abs() <= bound * (1 + u) + u * want.abs() + tiny).all())


@pytest.mark.parametrize("T,k,E,N,K,bn", [(1, 2, 8, 256, 512, 16), (16, 2, 8, 2048, 256, 16), (23, 6, 32, 200, 768, 32)])
def test_sums(T, k, E, N, K, bn):
    from vllm_b200.ops import cuda as cu
    R = T * k
    x, w, ids, offs, exact, bound = _case(R, N, K, E, torch.bfloat16, False, T)
    g = torch.Generator(device="cuda").manual_seed(T)
    pairs = torch.randperm(R, device="cuda", generator=g).int()
    pw = torch.rand(R, device="cuda", generator=g)
    acc = torch.zeros(T, N, device="cuda")
    cu.gemm_experts(x, w, offs, bn, None, (acc.data_ptr(), pairs, pw, k))
    tok, wt = pairs.long() // k, pw.double()[pairs.long()][:, None]
    want = torch.zeros(T, N, device="cuda", dtype=torch.double).index_add_(0, tok, exact * wt)
    size = torch.zeros_like(want).index_add_(0, tok, (exact.abs() + bound) * wt)
    room = torch.zeros_like(want).index_add_(0, tok, bound * wt) + (k + 1) * 2.0 ** -24 * size
    assert bool(((acc.double() - want).abs() <= room * 1.0001).all())
