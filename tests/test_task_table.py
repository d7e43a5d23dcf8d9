"""The table of attention tasks (ma_stage_tasks, ma_plan_set_tasks): its words against the numpy
statement of the schedule, and on the GPU the same result with and without it."""
import ctypes as C

import numpy as np
import pytest
import torch

from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.runtime import FusedFaOprojArWorkspace
from megaattention_b200.runtime.workspace import claim_order


def _stage(meta, prime, max_tasks, off=None):
    R, nb = meta.num_row_tiles, meta.num_batch
    offs = [int(x) for x in np.cumsum([0, nb + 1, nb + 1, R, R, R])]
    off = (offs[-1] + 6 + 3) // 4 * 4 if off is None else off
    buf = np.full(off + 4 + _cabi.TASK_WORDS * R + 1, -9, dtype=np.int32)
    a = _cabi.StageTasksArgs(_cabi.StageMetaArgs(
        meta.cu_seqlens_q.ctypes.data, meta.cu_seqlens_k.ctypes.data, meta.batch_idx.ctypes.data,
        meta.m_block.ctypes.data, buf.ctypes.data, nb, R, 4096, 8, 8, 1, 0, 0, prime, *offs, 0), off, max_tasks)
    return _cabi.lib.ma_stage_tasks(C.byref(a)), buf, off


@pytest.mark.parametrize("prime", [0, -1, 2])
@pytest.mark.parametrize("q,k", [([1], [1]), ([129, 128, 127, 1], [4000, 128, 300, 1]), ([700, 5, 2100], [700, 900, 2100])])
def test_the_table_says_what_the_arrays_say(q, k, prime):
    meta = build_row_desc(q, seqlens_k=k)
    R = meta.num_row_tiles
    rc, buf, off = _stage(meta, prime, R)
    assert rc == _cabi.MA_OK and buf[off:off + 4].tolist() == [R, 0, 0, 0] and buf[-1] == -9
    rows = buf[off + 4:off + 4 + _cabi.TASK_WORDS * R].reshape(R, -1)
    for row, t in zip(rows.tolist(), claim_order(meta, prime).tolist()):
        b = int(meta.batch_idx[t])
        assert row == [t, b, int(meta.m_block[t]), int(meta.cu_seqlens_q[b]), q[b], int(meta.cu_seqlens_k[b]), k[b], 0]


def test_a_table_that_is_too_small_or_misaligned_is_refused():
    meta = build_row_desc([300])
    assert _stage(meta, 0, 2)[0] == _cabi.MA_ERR_CAPACITY
    assert _stage(meta, 0, 3, off=22)[0] == _cabi.MA_ERR_INVALID


@pytest.mark.gpu
@pytest.mark.parametrize("paged", [False, True])
def test_with_and_without_the_table_are_the_same(paged):
    q, k = [257, 1, 128, 600], [900, 130, 128, 600]
    meta = build_row_desc(q, seqlens_k=k)
    kw = dict(paged=True, max_num_pages=32, max_num_pages_per_seq=8) if paged else {}
    ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, 384, 4, 128, q_per_kv=4, max_num_batch=4,
                                        max_tot_k=sum(k), device=torch.device("cuda:0"), **kw).compile()
    g = torch.Generator().manual_seed(3)
    t = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)      # noqa: E731
    if paged:
        kv, extra = (t(32, 128, 1, 128), t(32, 128, 1, 128)), (torch.arange(32, dtype=torch.int32).view(4, 8),
                                                               torch.tensor(k, dtype=torch.int32))
    else:
        kv, extra = (t(sum(k), 1, 128), t(sum(k), 1, 128)), ()
    ws.set_layer(meta, t(sum(q), 4, 128), *kv, t(512, 384), *extra)
    out = []
    for table in (ws.tasks.data_ptr(), 0):
        _cabi.check(ws._lib.ma_plan_set_tasks(ws._plan, table), "ma_plan_set_tasks")
        ws.csym.zero_()
        ws.launch()
        ws.check_status()
        out.append(ws.output().clone())
    assert torch.equal(*out) and out[0].abs().max() > 0
    assert ws._lib.ma_plan_set_tasks(ws._plan, ws.tasks.data_ptr() + 4) == _cabi.MA_ERR_INVALID
