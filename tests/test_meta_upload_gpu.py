"""A step's metadata on the device (ma_upload_meta): every array's active part, and nothing else,
for steps that fit the small parameter block, the large one, and several of those."""
import numpy as np
import pytest
import torch

from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.metadata.row_desc import active_counts
from megaattention_b200.runtime import FusedFaOprojArWorkspace
from megaattention_b200.runtime.workspace import claim_order

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [[1], [128] * 72, [128] * 73, [64000, 5], [128] * 300, [100000, 1]])
def test_what_is_uploaded(q):
    meta = build_row_desc(q)
    R, nb = meta.num_row_tiles, meta.num_batch
    ws = FusedFaOprojArWorkspace.create(None, R + 3, 128, 2, 128, max_num_batch=nb + 2, max_tot_k=sum(q),
                                        device=torch.device("cuda:0"))
    ws.meta_dev.fill_(-7)
    ws.set_meta(meta)
    order = claim_order(meta, 0)
    parts = [(ws.cu_q, meta.cu_seqlens_q), (ws.cu_k, meta.cu_seqlens_k), (ws.fa_b, meta.batch_idx),
             (ws.fa_mb, meta.m_block), (ws.actv, active_counts(R, 2, ws.num_super_groups, 1, 0))]
    for got, want in parts:
        assert got[:len(want)].tolist() == want.tolist() and (got[len(want):] == -7).all()
    got = ws.fa_order.tolist()
    assert got[:R] in (order.tolist(), claim_order(meta, -1).tolist()) and set(got[R:]) <= {-7}
    table = ws.tasks.cpu().numpy()
    assert table[:4].tolist() == [R, 0, 0, 0] and (table[4 + _cabi.TASK_WORDS * R:] == -7).all()
    assert table[4:4 + _cabi.TASK_WORDS * R].reshape(R, -1)[:, 0].tolist() == got[:R]
    # a later, smaller step leaves no trace of the arrays' staging in its own words
    small = build_row_desc([min(q[0], 130)])
    ws.set_meta(small)
    assert ws.cu_q[:2].tolist() == small.cu_seqlens_q.tolist() and ws.tasks[0].item() == small.num_row_tiles
    assert np.array_equal(ws.fa_b[:small.num_row_tiles].cpu().numpy(), small.batch_idx)
