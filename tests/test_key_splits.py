"""Row tiles whose keys are split into parts (ma_stage_tasks, ma_plan_set_split): what the task table
says of them, and on the GPU the result against the oracle and against whole tasks."""
import ctypes as C
import heapq
import time

import numpy as np
import pytest
import torch

from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.runtime import FusedFaOprojArWorkspace
from oracle.chain_oracle import err_beyond_rounding, full_chain_oracle


def _staged(q, k, heads, ctas, slots, room, prime):
    meta = build_row_desc(q, seqlens_k=k)
    R, nb = meta.num_row_tiles, meta.num_batch
    offs = [int(x) for x in np.cumsum([0, nb + 1, nb + 1, R, R, R])]
    off = (offs[-1] + 6 + 3) // 4 * 4
    room = R + slots if room is None else room
    buf = np.full(off + 4 + _cabi.TASK_WORDS * room + 1, -9, dtype=np.int32)
    a = _cabi.StageTasksArgs(_cabi.StageMetaArgs(
        meta.cu_seqlens_q.ctypes.data, meta.cu_seqlens_k.ctypes.data, meta.batch_idx.ctypes.data,
        meta.m_block.ctypes.data, buf.ctypes.data, nb, R, 4096, heads, 8, 1, 0, 0, prime, *offs, 0),
        off, room, slots, ctas)
    return a, buf, meta


def _table(q, k, heads, ctas=148, slots=80, room=None, prime=0):
    a, buf, meta = _staged(q, k, heads, ctas, slots, room, prime)
    off = a.off_tasks
    assert _cabi.lib.ma_stage_tasks(C.byref(a)) == _cabi.MA_OK and buf[-1] == -9
    n = int(buf[off])
    rows = buf[off + 4:off + 4 + _cabi.TASK_WORDS * n].reshape(n, -1)
    nblk = [min(-(-k[b] // 128), -(-((m + 1) * 128 + k[b] - q[b]) // 128))
            for b, m in zip(meta.batch_idx.tolist(), meta.m_block.tolist())]
    return rows, nblk


def _check(rows, nblk, slots):
    """Every part of every row tile once, no slot twice, claimed longest first; the parts' lengths."""
    got, used, lens = {}, set(), []
    for r in rows:
        s = int(np.uint32(r[7]))
        n, part, first = max(s & 255, 1), s >> 8 & 255, s >> 16
        got.setdefault(int(r[0]), []).append((n, part))
        t = nblk[int(r[0])]
        lens.append(t * (part + 1) // n - t * part // n)
        if n > 1:
            assert first + part not in used and first + part < slots and n <= 16
            used.add(first + part)
    assert sorted(got) == list(range(len(nblk)))
    for parts in got.values():
        assert sorted(p for _, p in parts) == list(range(parts[0][0])) and len({n for n, _ in parts}) == 1
    return lens


@pytest.mark.parametrize("q,k,heads,split", [
    ([2000], [15871], 8, True),                       # few tasks, all long
    ([17, 256, 45, 1], [2065, 3300, 801, 5217], 8, True),     # one much longer than the rest
    ([1], [30000], 1, True), ([1], [30000], 64, True), ([300], [2500], 7, True),
    ([128], [1152], 8, False),                        # 9 key blocks: two parts would be too short
    ([1024] * 4, None, 16, False), ([16384], None, 8, False),     # enough tasks
    ([7500, 4100, 3300, 2600, 2000, 1500, 1000, 600], None, 16, False),
])
def test_what_is_split(q, k, heads, split):
    k = q if k is None else k
    slots = 640 // heads
    rows, nblk = _table(q, k, heads, slots=slots)
    lens = _check(rows, nblk, slots)
    assert (len(rows) > len(nblk)) == split
    assert lens == sorted(lens, reverse=True)
    if split:
        assert max(lens) < max(nblk) and min(lens) >= min(3, min(nblk))
    assert len(_table(q, k, heads, slots=0)[0]) == len(nblk)          # no room, no parts


def test_splits_keep_to_the_room_there_is():
    q, k = [2000], [15871]
    for slots in (2, 16, 31, 32, 47):
        rows, nblk = _table(q, k, 8, slots=slots)
        _check(rows, nblk, slots)
        rows, nblk = _table(q, k, 8, slots=80, room=len(nblk) + slots)
        assert len(rows) <= len(nblk) + slots
    rows, nblk = _table(q, k, 8, prime=-1)
    _check(rows, nblk, 80)
    assert len(rows) > len(nblk)


@pytest.mark.parametrize("seed", range(40))
def test_drawn_batches(seed):
    rng = np.random.RandomState(seed)
    n = int(np.exp(rng.uniform(0, np.log(24))))
    q = [int(x) for x in np.exp(rng.uniform(0, np.log(3000), n)).astype(int) + 1]
    k = [a + int(rng.uniform(0, 12000)) for a in q]
    heads = int(rng.choice([1, 2, 3, 4, 7, 8, 16, 64]))
    slots = 640 // heads
    rows, nblk = _table(q, k, heads, ctas=int(rng.choice([1, 5, 148])), slots=slots)
    _check(rows, nblk, slots)


def _parts(nblk, heads, hidden, ctas, slots):
    """The model that csrc/meta.cpp chooses by, candidate by candidate and task by task."""
    lanes, most = max(1, ctas // ((heads + 1) // 2)), max(nblk)
    whole = [1] * len(nblk)
    if slots < 2 or most < 10 or len(nblk) * ((heads + 1) // 2) > 3 * ctas:
        return whole
    oproj = 0.2 * len(nblk) * -(-hidden // 128) * heads / ctas

    def takes(costs):
        busy = [0] * lanes
        for c in sorted(costs, reverse=True):
            heapq.heapreplace(busy, busy[0] + c)
        return max(max(busy), sum(costs) / lanes + oproj)

    if most + 2 <= sum(n + 2 for n in nblk) / lanes + oproj:
        return whole
    best, parts = 0.9 * takes([n + 2 for n in nblk]), whole
    for k in range(2, min(16, most // 5) + 1):
        split = [-(-n // -(-most // k)) for n in nblk]
        if sum(m for m in split if m > 1) > slots:
            break
        t = takes([n * (i + 1) // m - n * i // m + 2 + (m > 1)
                   for n, m in zip(nblk, split) for i in range(m)]) + 0.5 * k
        if t < best:
            best, parts = t, split
    return parts


def _prefixed(seed, most_keys=12000):
    rng = np.random.RandomState(seed)
    n = int(np.exp(rng.uniform(0, np.log(24))))
    q = [int(x) for x in np.exp(rng.uniform(0, np.log(3000), n)).astype(int) + 1]
    return q, [a + int(rng.uniform(0, most_keys)) for a in q], rng


@pytest.mark.parametrize("heads", [1, 2, 3, 8, 16, 64])
def test_the_parts_are_the_models(heads):
    split = 0
    for seed in range(40):
        q, k, rng = _prefixed(seed, 60000 if seed % 4 == 0 else 12000)
        ctas, slots = int(rng.choice([1, 7, 148, 148])), int(rng.choice([640 // heads, 640 // heads, 9]))
        rows, nblk = _table(q, k, heads, ctas=ctas, slots=slots)
        got = np.bincount(rows[:, 0], minlength=len(nblk)).tolist()
        assert got == _parts(nblk, heads, 4096, ctas, slots), (seed, q, k, ctas, slots)
        split += max(got) > 1
    assert split >= 3


def test_the_choice_is_a_small_part_of_a_steps_host_time():
    """It runs in every call, a paged call's while the GPU waits: with few heads there are many tasks and
    many lanes to look at.  (One candidate after the other, each with all of its tasks sorted and
    simulated: 30 times the rest of ma_stage_tasks; now 4.)"""
    args = []
    for seed in range(24):
        q, k, _ = _prefixed(seed)
        args.append((_staged(q, k, 1, 148, 640, None, 0), _staged(q, k, 1, 148, 0, None, 0)))

    def spent(a):
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            _cabi.lib.ma_stage_tasks(C.byref(a))
            t.append(time.perf_counter() - t0)
        return min(t)

    with_parts, without = (sum(spent(a[i][0]) for a in args) for i in (0, 1))
    assert with_parts < 12 * without, (with_parts, without)


def _inputs(q, k, heads, kv, hidden):
    g = torch.Generator().manual_seed(11)
    t = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)      # noqa: E731
    W = (t(heads * 128, hidden).float() * (heads * 128) ** -0.5).to(torch.bfloat16)
    return t(sum(q), heads, 128), t(sum(k), kv, 128), t(sum(k), kv, 128), W


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv", [(8, 1), (1, 1), (3, 3), (7, 1)])
@pytest.mark.parametrize("q,k", [([130, 1, 40], [4000, 2049, 300]), ([257], [2305])])
def test_parts_against_the_oracle_and_whole_tasks(q, k, heads, kv):
    hidden = 384
    meta = build_row_desc(q, seqlens_k=k)
    Q, K, V, W = _inputs(q, k, heads, kv, hidden)
    ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, hidden, heads, 128, q_per_kv=heads // kv,
                                        max_num_batch=len(q), max_tot_k=sum(k), device=torch.device("cuda:0"))
    _, Yp, _ = full_chain_oracle(Q, K, V, W, q, k)
    outs = []
    for audit in (False, True):
        ws.compile(audit=audit)
        for _ in range(3):                       # (the counts of parts start from zero each time)
            ws.csym.fill_(-7.0)
            ws.set_layer(meta, Q, K, V, W)
            ws.launch()
            ws.check_status()
            outs.append(ws.output().cpu())
        assert int(ws.tasks[0]) > meta.num_row_tiles and not ws.part_count.any() and not any(ws.ctrl.tolist())
        if audit:
            fa, op, _ = ws.audit_counts()
            assert (fa == 3).all() and (op == 3).all()
    assert all(torch.equal(o, outs[0]) for o in outs)      # whoever is last adds the same sum
    assert err_beyond_rounding(outs[0], Yp) <= 8e-3
    # whole tasks of the same table (no room for parts): the same to the rounding of P and O
    _cabi.check(ws._lib.ma_plan_set_split(ws._plan, 0, 0), "ma_plan_set_split")
    ws.launch()
    ws.check_status()
    whole = ws.output().cpu()
    assert not torch.equal(whole, outs[0]) and err_beyond_rounding(whole, Yp) <= 8e-3
    assert ws._lib.ma_plan_set_split(ws._plan, ws.parts.data_ptr(), 0) == _cabi.MA_ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[4000, 3000], [900, 640], [130, 64]])
def test_paged_lengths_on_the_device_decide(lens):
    """The host split by lengths of 4000 and 3000 keys; the device's may be shorter than the parts."""
    q, most, heads, hidden = [130, 33], [4000, 3000], 8, 256
    meta = build_row_desc(q, seqlens_k=most)
    Q, K, V, W = _inputs(q, lens, heads, 1, hidden)
    ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, hidden, heads, 128, q_per_kv=heads, paged=True,
                                        max_num_batch=2, max_tot_k=8192, max_num_pages=64, max_num_pages_per_seq=32,
                                        device=torch.device("cuda:0")).compile()
    table = torch.arange(64, dtype=torch.int32).view(2, 32).flip(0)
    kc, vc = torch.zeros(64, 128, 1, 128, dtype=torch.bfloat16), torch.zeros(64, 128, 1, 128, dtype=torch.bfloat16)
    at = 0
    for b, n in enumerate(lens):
        for cache, src in ((kc, K), (vc, V)):
            cache.view(-1, 1, 128)[int(table[b, 0]) * 128:][:n] = src[at:at + n]
        at += n
    ws.set_layer(meta, Q, kc, vc, W, page_table=table, cache_seqlens=torch.tensor(lens, dtype=torch.int32))
    ws.launch()
    ws.check_status()
    assert int(ws.tasks[0]) > meta.num_row_tiles and not ws.part_count.any()
    _, Yp, _ = full_chain_oracle(Q, K, V, W, q, lens)
    assert err_beyond_rounding(ws.output().cpu(), Yp) <= 8e-3


@pytest.mark.gpu
def test_a_workspace_without_room_for_parts():
    q, k, heads, hidden = [130, 1, 40], [4000, 2049, 300], 8, 384
    meta = build_row_desc(q, seqlens_k=k)
    Q, K, V, W = _inputs(q, k, heads, 1, hidden)
    out = []
    for room in (True, False):
        ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, hidden, heads, 128, q_per_kv=heads,
                                            max_num_batch=len(q), max_tot_k=sum(k), device=torch.device("cuda:0"),
                                            key_splits=room).compile()
        ws.set_layer(meta, Q, K, V, W)
        ws.launch()
        ws.check_status()
        assert (int(ws.tasks[0]) > meta.num_row_tiles) == room and bool(ws.parts.numel()) == room
        out.append(ws.output().cpu())
    _, Yp, _ = full_chain_oracle(Q, K, V, W, q, k)
    assert all(err_beyond_rounding(o, Yp) <= 8e-3 for o in out)
