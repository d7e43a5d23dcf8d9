"""The O_proj task shapes of a single rank (row tiles x column tiles: 2 x 2, 1 x 2, 1 x 1,
chosen by the number of 2 x 2 tasks per CTA) against the oracle: odd numbers of row tiles and
of column tiles, a partial row tile in either half of a pair, a hidden size that ends inside
a tile.  The CTA count picks the shape; the audit build says which one ran."""
import pytest
import torch

from test_fused_single_gpu import _case_inputs, check, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ctas,shape", [
    ("c1", 1, (2, 2)), ("c1", 4, (2, 2)), ("c1", 5, (2, 2)), ("c1", 6, (1, 2)), ("c1", 8, (1, 2)), ("c1", 148, (1, 1)),
    ("ragged_hidden", 2, (2, 2)), ("ragged_hidden", 4, (1, 2)), ("ragged_hidden", 6, (1, 1)),
    ("multi_seq", 1, (2, 2)), ("multi_seq", 3, (1, 2)),
    ("vm44_300", 1, (1, 2)), ("gqa_q4_vm44", 1, (1, 2)), ("gqa_q4_vm44", 2, (1, 1)),
])
def test_task_shapes(name, ctas, shape):
    res = run_case(name, num_ctas=ctas, launches=3, audit=True)
    assert res["op_shape"] == shape
    check(res)
    check(run_case(name, num_ctas=ctas, launches=2))


def _launched(sq, H, hidden, qpk, sk, inputs, sg, ctas, audit):
    from megaattention_b200.metadata import build_row_desc
    from megaattention_b200.runtime import FusedFaOprojArWorkspace
    meta = build_row_desc(sq, seqlens_k=sk)
    ws = FusedFaOprojArWorkspace.create(
        None, max_num_row_tiles=meta.num_row_tiles, hidden=hidden, H_local=H, D=128, q_per_kv=qpk,
        super_group_n_tiles=sg, max_tot_k=int(meta.cu_seqlens_k[-1]), device="cuda:0")
    ws.compile(w_fa=2, w_oproj=1, w_ar=0, num_ctas=ctas, audit=audit)
    ws.set_layer(meta, *(x.cuda() for x in inputs))
    ws.launch()
    ws.check_status()
    return ws


@pytest.mark.parametrize("name", ["c1", "ragged_hidden", "multi_seq", "gqa_q4_vm44"])
@pytest.mark.parametrize("sg", [1, 3, 4])
def test_slot_tasks_of_several_ranks(name, sg):
    """With MA_FLAG_NO_AR a single rank runs the tasks that several ranks have (one row tile x
    `sg` column tiles in passes of two): the same bits as its own task shapes give."""
    from megaattention_b200 import _cabi
    (sq, H, hidden, qpk, sk, _), inputs = _case_inputs(name)
    ws = _launched(sq, H, hidden, qpk, sk, inputs, sg, 3, False)
    want = ws.csym.clone()
    ws.csym.zero_()
    for _ in range(2):
        ws.launch(flags=_cabi.MA_FLAG_NO_AR)
    ws.check_status()
    assert torch.equal(ws.csym.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("ctas,shape", [(1, (2, 2)), (24, (2, 2)), (25, (1, 2)), (48, (1, 2)), (49, (1, 1)),
                                        (148, (1, 1))])
def test_shapes_of_the_stage_alone(ctas, shape):
    """O_proj-only launches have lines of their own (12 2 x 2 tasks here: half and a quarter of a
    wave); 8 heads, so that a task goes round its ring of stages several times.  The same bits
    as the whole launch, every time."""
    from cases import _randn
    sq, H, hidden = [300, 100, 120], 8, 900               # 5 row tiles x 8 column tiles
    n = sum(sq)
    inputs = (_randn((n, H, 128), 5100), _randn((n, 1, 128), 5101), _randn((n, 1, 128), 5102),
              _randn((H * 128, hidden), 5103, float(H * 128) ** -0.5))
    ws = _launched(sq, H, hidden, H, None, inputs, 4, ctas, True)
    want = ws.csym.clone()
    for _ in range(2):
        ws.csym.zero_()
        ws.launch_oproj_only()
        ws.check_status()
        assert tuple(ws.status.cpu().tolist()[6:8]) == shape
        assert torch.equal(ws.csym.view(torch.int16), want.view(torch.int16))
