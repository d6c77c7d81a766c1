"""The gated delta rule from raw projections: heads in groups, odd widths, edges of the staged chunks, strong decays, states that go on."""
import pytest
import torch
import torch.nn.functional as F

from vllm_b200.forward_context import AttentionMetadata

pytestmark = pytest.mark.gpu


def _oracle(qkvz, ba, cw, A_log, dt_bias, norm_w, conv0, S0, nk, nv, dk, dv, beta_scale, eps):
    """One request in 64 bits: (gated output [T, nv * dv], window, state)."""
    T, r = qkvz.shape[0], nv // nk
    q, k, v, z = qkvz.view(T, nk, -1).split([dk, dk, r * dv, r * dv], -1)
    b, a = ba.view(T, nk, 2 * r).split([r, r], -1)
    x = torch.cat([conv0.t(), torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], -1)])
    K = cw.shape[1]
    c = F.silu(sum(x[i:i + T] * cw[:, i] for i in range(K)))
    q, k, v = c.split([nk * dk, nk * dk, nv * dv], -1)
    unit = lambda y: (y.view(T, nk, dk) * torch.rsqrt(y.view(T, nk, dk).pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(r, 1)  # noqa: E731
    q, k, v = unit(q) * dk ** -0.5, unit(k), v.view(T, nv, dv)
    g = (-A_log.exp() * F.softplus(a.reshape(T, nv) + dt_bias)).exp()
    beta, S, out = b.reshape(T, nv).sigmoid() * beta_scale, S0.clone(), []
    for t in range(T):
        S = S * g[t, :, None, None]
        d = (v[t] - torch.einsum("hkv,hk->hv", S, k[t])) * beta[t, :, None]
        S = S + k[t, :, :, None] * d[:, None]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]))
    o = torch.stack(out)
    o = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + eps) * norm_w * F.silu(z.reshape(T, nv, dv))
    return o.reshape(T, -1), x[T:].t(), S


@pytest.mark.parametrize("nk,nv,dk,dv", [(2, 4, 128, 256), (3, 3, 64, 40), (1, 2, 32, 66), (2, 2, 256, 72), (1, 1, 96, 64), (2, 2, 160, 16)])
@pytest.mark.parametrize("decay", [0.0, 4.0])
def test_against_recurrence(nk, nv, dk, dv, decay):
    from vllm_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s, scale=1.0: torch.randn(*s, device="cuda", generator=g) * scale  # noqa: E731
    bf = torch.bfloat16
    q_lens, ctx = [1, 7, 8, 9, 33, 1], [0, 0, 3, 5, 0, 12]
    r, K, T = nv // nk, 4, sum(q_lens)
    C = 2 * nk * dk + nv * dv
    group, off = 2 * dk + 2 * r * dv, C * (K - 1)
    qkvz, ba = rnd(T, nk * group).to(bf), rnd(T, 2 * nv).to(bf)
    cw, A_log, dt_bias, norm_w = rnd(C, K, scale=0.5).to(bf), rnd(nv) * 0.5 + decay, rnd(nv), (1 + 0.1 * rnd(dv)).to(bf)
    n = len(q_lens)
    pool = rnd(n + 2, off + nv * dk * dv + (-(off + nv * dk * dv)) % 4, scale=0.3)
    pool[:, :off] = pool[:, :off].to(bf).float()               # windows hold inputs of the model's type
    rows = torch.randperm(n + 2, device="cuda", generator=g)[:n].int()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    cu_q = [sum(q_lens[:i]) for i in range(n + 1)]
    md = AttentionMetadata(num_reqs=n, num_actual_tokens=T, max_query_len=max(q_lens), max_seq_len=64, query_start_loc=i32(cu_q),
                           seq_lens=i32([a + b for a, b in zip(q_lens, ctx)]), block_table=rows[:, None].contiguous(), slot_mapping=None)
    want = []
    for i in range(n):
        st = pool[rows[i].long()].double() * (ctx[i] > 0)
        sl = slice(cu_q[i], cu_q[i + 1])
        want.append(_oracle(qkvz[sl].double(), ba[sl].double(), cw.double(), A_log.double(), dt_bias.double(), norm_w.double(),
                            st[:off].view(C, K - 1), st[off:off + nv * dk * dv].view(nv, dk, dv), nk, nv, dk, dv, 2.0, 1e-5))
    conv = cu.causal_conv1d(qkvz, cw, None, pool, md, heads=(group, nk, dk, r * dv))
    o = cu.gated_delta(conv, ba, A_log, dt_bias, pool, off, md, nk, nv, dk, dv, 2.0, 1e-6)
    y = cu.gated_norm(o, qkvz[:, 2 * dk + r * dv:], norm_w, nv, 1e-5, False, z_heads=(nv * dv, r, group))
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    assert rel(y, torch.cat([w[0] for w in want])) < 2 ** -8.5          # one rounding to 16 bits; 32-bit sums of dk products before it
    for i in range(n):
        st = pool[rows[i].long()]
        assert rel(st[off:off + nv * dk * dv].view(nv, dk, dv), want[i][2]) < 2e-5
        assert torch.equal(st[:off].view(C, K - 1).double(), want[i][1])
