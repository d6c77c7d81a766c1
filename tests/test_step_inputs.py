"""Rows of the device tables follow the runner's batch: moves, admissions and appended blocks of a step as one packed list."""
import random

import numpy as np
import pytest
import torch

from vllm_b200.worker.model_runner import ModelRunner, ReqState, _Staging


def _runner(R, L, MB, G):
    r = object.__new__(ModelRunner)
    r.max_num_reqs, r.num_kv_groups, r.gpu_prep, r.is_cuda = R, G, True, False
    r.req_ids, r.req_index, r.states, r._parked, r.cross_states = [], {}, {}, {}, {}
    r.token_ids_cpu = np.zeros((R, L), dtype=np.int32)
    for n in ("num_tokens_cpu", "num_logical_cpu", "num_prompt_cpu", "num_computed_cpu", "temp_cpu", "seed_cpu", "mode_cpu", "lp_cpu", "filter_cpu"):
        setattr(r, n, np.zeros(R, dtype=np.int64))
    r.block_tables_cpu = [np.zeros((R, MB), dtype=np.int32) for _ in range(G)]
    r.num_blocks_cpu = [np.zeros(R, dtype=np.int32) for _ in range(G)]
    r._bt_diffs, r._new_tokens, r._row_at, r._late_rows = [[] for _ in range(G)], [], {}, []
    return r


def _apply(v, tables, launches):
    """What the device does with the list."""
    for at, n, which, moved in launches:
        tbl, row, start, cnt, off = v[at:at + 5 * n].reshape(5, n)
        before = [t.copy() for t in tables]
        for e in range(n):
            t = which * 9 + tbl[e]
            src = before[t][off[e]] if moved else v[off[e]:]
            tables[t][row[e], start[e]:start[e] + cnt[e]] = src[:cnt[e]]


@pytest.mark.parametrize("G", [1, 2, 9, 20])
@pytest.mark.parametrize("room", [None, 60])         # 60 behind the moves: most changes do not fit and go late
def test_rows_follow_the_batch(G, room):
    R, L, MB = 8, 40, 6
    rng, r = random.Random(G), _runner(8, 40, 6, G)
    stg = _Staging(64, R, MB, G, False)
    stg.room = 5 * R * (4 + 6 * G) + 64 + G * R * MB if room is None else 5 * R * (1 + G) + room
    stg.np_pack = np.zeros(8 * R + stg.room, dtype=np.int32)
    dev = [np.zeros((R, L), dtype=np.int32)] + [np.zeros((R, MB), dtype=np.int32) for _ in range(G)]
    n = 0
    for step in range(300):
        for _ in range(rng.randint(0, 2)):           # (steps without a flush between them compose)
            gone = rng.sample(r.req_ids, rng.randint(0, len(r.req_ids)))
            for rid in sorted(gone, key=lambda x: r.req_index[x], reverse=rng.random() < 0.8):
                r._remove(rid)
            while len(r.req_ids) < R and rng.random() < 0.6:
                n += 1
                st = ReqState(str(n), -1, None, None, None)
                r._add_row(st, [n * 100 + i for i in range(rng.randint(1, L - 20))],
                           [[n * 50 + g + i for i in range(rng.randint(1, MB - 3))] for g in range(G)], 0)
            for rid in r.req_ids:
                row = r.req_index[rid]
                for g in range(G):
                    k = r.num_blocks_cpu[g][row]
                    if k < MB and rng.random() < 0.2:
                        r.block_tables_cpu[g][row, k] = rng.randint(1, 10 ** 6)
                        r.num_blocks_cpu[g][row] = k + 1
                        r._bt_diffs[g].append((rid, int(k), [int(r.block_tables_cpu[g][row, k])]))
        end, launches = r._pack_gpu_state(stg)
        assert end <= len(stg.np_pack) and not r._row_at and not any(r._bt_diffs)
        _apply(stg.np_pack, dev, launches)
        for t, row in r._late_rows:
            k = r.num_tokens_cpu[row] if t == 0 else r.num_blocks_cpu[t - 1][row]
            dev[t][row, :k] = (r.token_ids_cpu if t == 0 else r.block_tables_cpu[t - 1])[row, :k]
        r._late_rows.clear()
        for rid in r.req_ids:
            row = r.req_index[rid]
            k = r.num_tokens_cpu[row]
            if rng.random() < 0.7:                   # the step appends a token on the device, the host learns of it
                tok = rng.randint(1, 10 ** 6)
                if k < L:
                    dev[0][row, k] = r.token_ids_cpu[row, k] = tok
                    r.num_tokens_cpu[row] = r.num_logical_cpu[row] = k = k + 1
            assert np.array_equal(dev[0][row, :k], r.token_ids_cpu[row, :k])
            for g in range(G):
                k = r.num_blocks_cpu[g][row]
                assert np.array_equal(dev[1 + g][row, :k], r.block_tables_cpu[g][row, :k]), (step, rid, g)


@pytest.mark.gpu
@pytest.mark.parametrize("G", [1, 2, 8, 11])
@pytest.mark.parametrize("nb,pad_b,pad_t", [(1, 1, 0), (5, 8, 0), (33, 40, 300), (40, 40, 0)])
def test_one_launch_serves_all_groups(G, nb, pad_b, pad_t):
    from vllm_b200.ops import cuda_ops
    cu, R, L, MB, BS = cuda_ops(), 48, 256, 8, 32
    rng = np.random.default_rng(nb + G)
    t = lambda a: torch.tensor(np.asarray(a), device="cuda")                      # noqa: E731
    tokens = torch.randint(0, 9999, (R, L), dtype=torch.int32, device="cuda")
    rows_of = [torch.randint(1, 999, (R, MB), dtype=torch.int32, device="cuda") for _ in range(G)]
    rows, nc = rng.permutation(R)[:nb].astype(np.int32), rng.integers(0, 200, nb).astype(np.int32)
    ns = rng.integers(1, 6, nb).astype(np.int32) if pad_t else np.ones(nb, dtype=np.int32)

    def buffers():
        n = 512
        return dict(ids=torch.full((n,), 7, dtype=torch.int32, device="cuda"), pos=torch.full((n,), 7, dtype=torch.int64, device="cuda"),
                    qsl=torch.full((pad_b + 1,), 7, dtype=torch.int32, device="cuda"), sl=torch.full((pad_b,), 7, dtype=torch.int32, device="cuda"),
                    slots=[torch.full((n,), 7, dtype=torch.int64, device="cuda") for _ in range(G)],
                    bt=[torch.full((pad_b, MB), 7, dtype=torch.int32, device="cuda") for _ in range(G)])
    a, b = buffers(), buffers()
    meta = [t(rows), t(nc), t(ns)]
    last = torch.full((pad_b,), -7, dtype=torch.int64, device="cuda")
    cu.prep_step_groups(*[m.data_ptr() for m in meta], nb, tokens, G, cu.pointers(rows_of), MB, a["ids"], a["pos"], a["qsl"], a["sl"], last,
                        cu.pointers(a["slots"]), cu.pointers(a["bt"]), MB, 7, BS, pad_b, pad_t)
    for g in range(G):                                                            # group by group
        cu.prep_step(*meta, tokens, rows_of[g], b["ids"], b["pos"], b["qsl"], b["sl"], b["slots"][g], b["bt"][g], 7, BS, pad_b=pad_b, pad_t=pad_t,
                     write_tokens=g == 0)
    for k in ("ids", "pos", "qsl", "sl"):
        assert torch.equal(a[k], b[k])
    for g in range(G):
        assert torch.equal(a["slots"][g], b["slots"][g]) and torch.equal(a["bt"][g], b["bt"][g])
    assert last[:nb].tolist() == (np.cumsum(ns) - 1).tolist() and (last[nb:] == -7).all()


@pytest.mark.gpu
@pytest.mark.parametrize("nb,cols", [(1, 0), (1, 3), (64, 13), (700, 131)])
def test_results_reach_tables_and_host(nb, cols):
    from vllm_b200.ops import cuda_ops
    cu, L = cuda_ops(), 16
    table = torch.zeros(nb + 3, L, dtype=torch.int32, device="cuda")
    rows = torch.randperm(nb + 3, device="cuda")[:nb].int()
    pos = torch.randint(-1, L, (nb,), device="cuda").int()
    ids = torch.randint(0, 99999, (nb,), device="cuda")
    host = torch.full((nb + 2,), -5, dtype=torch.int64).pin_memory()
    lp = torch.randint(-2 ** 31, 2 ** 31 - 1, (nb, cols), device="cuda").int() if cols else None
    host_lp = torch.zeros(nb, cols, dtype=torch.int32).pin_memory() if cols else None
    cu.publish(table, rows.data_ptr(), pos.data_ptr(), ids, nb, host, lp, host_lp)
    ev = torch.cuda.Event()
    ev.record()
    ev.synchronize()
    assert torch.equal(host[:nb], ids.cpu()) and (host[nb:] == -5).all()
    assert lp is None or torch.equal(host_lp, lp.cpu())
    want = torch.zeros_like(table)
    for r, p, i in zip(rows.tolist(), pos.tolist(), ids.tolist()):
        if p >= 0:
            want[r, p] = i
    assert torch.equal(table, want)
