"""The O_proj task shapes of a single rank (row tiles x column tiles: 2 x 2, 1 x 2, 1 x 1,
chosen by the number of 2 x 2 tasks per CTA) against the oracle: odd numbers of row tiles and
of column tiles, a partial row tile in either half of a pair, a hidden size that ends inside
a tile.  The CTA count picks the shape: with t 2 x 2 tasks, n CTAs, 2 x 2 from t >= 3 n, two
column tiles from 4 t >= 5 n."""
import pytest
import torch

from test_fused_single_gpu import CASES, _case_inputs, check, run_case

pytestmark = pytest.mark.gpu


def _shape(name, ctas):
    sq, hidden = CASES[name][0], CASES[name][2]
    tiles, num_out = sum(-(-n // 128) for n in sq), -(-hidden // 128)
    t = -(-tiles // 2) * -(-num_out // 2)
    return (2 if t >= 3 * ctas else 1, 2 if 4 * t >= 5 * ctas else 1)


@pytest.mark.parametrize("name,ctas,shape", [
    ("c1", 1, (2, 2)), ("c1", 4, (2, 2)), ("c1", 8, (1, 2)), ("c1", 148, (1, 1)),
    ("ragged_hidden", 2, (2, 2)), ("ragged_hidden", 4, (1, 2)), ("ragged_hidden", 6, (1, 1)),
    ("multi_seq", 1, (2, 2)), ("multi_seq", 3, (1, 2)),
    ("vm44_300", 1, (1, 2)), ("gqa_q4_vm44", 1, (1, 2)), ("gqa_q4_vm44", 2, (1, 1)),
])
def test_task_shapes(name, ctas, shape):
    assert _shape(name, ctas) == shape
    check(run_case(name, num_ctas=ctas, launches=3, audit=True))
    check(run_case(name, num_ctas=ctas, launches=2))


@pytest.mark.parametrize("name", ["c1", "ragged_hidden", "multi_seq", "gqa_q4_vm44"])
@pytest.mark.parametrize("sg", [1, 3, 4])
def test_slot_tasks_of_several_ranks(name, sg):
    """With MA_FLAG_NO_AR a single rank runs the tasks that several ranks have (one row tile x
    `sg` column tiles in passes of two): the same bits as its own task shapes give."""
    from megaattention_b200 import _cabi
    from megaattention_b200.metadata import build_row_desc
    from megaattention_b200.runtime import FusedFaOprojArWorkspace
    (sq, H, hidden, qpk, sk, _), (Q, K, V, W) = _case_inputs(name)
    meta = build_row_desc(sq, seqlens_k=sk)
    ws = FusedFaOprojArWorkspace.create(
        None, max_num_row_tiles=meta.num_row_tiles, hidden=hidden, H_local=H, D=128, q_per_kv=qpk,
        super_group_n_tiles=sg, max_tot_k=int(meta.cu_seqlens_k[-1]), device="cuda:0")
    ws.compile(w_fa=2, w_oproj=1, w_ar=0, num_ctas=3)
    ws.set_layer(meta, Q.cuda(), K.cuda(), V.cuda(), W.cuda())
    ws.launch()
    want = ws.csym.clone()
    ws.csym.zero_()
    for _ in range(2):
        ws.launch(flags=_cabi.MA_FLAG_NO_AR)
    ws.check_status()
    assert torch.equal(ws.csym.view(torch.int16), want.view(torch.int16))
