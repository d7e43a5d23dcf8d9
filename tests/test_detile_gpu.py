"""``ws.output()`` (csrc/detile.cu) against the tile-by-tile copy it stands for: bit for bit,
at the widths that take its three access sizes, with one row, full and ragged tiles, and more
sequences than one launch carries."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [1, 63, 130, 200, 1024, 2056])
@pytest.mark.parametrize("lens", [[1], [128], [129, 1, 300], [1 + (7 * i) % 40 for i in range(600)]])
def test_output_is_the_packed_copy(hidden, lens):
    from megaattention_b200.metadata import build_row_desc
    from megaattention_b200.runtime import FusedFaOprojArWorkspace
    meta = build_row_desc(lens)
    ws = FusedFaOprojArWorkspace.create(
        None, meta.num_row_tiles + 1, hidden, 1, 128, max_num_batch=len(lens),
        max_tot_k=sum(lens), device="cuda:0")
    ws.compile()
    ws.csym.normal_()
    got = ws.output(meta).cpu()
    flat = ws.csym.cpu().view(ws.max_num_row_tiles, 128, ws.hidden_pad)
    want = torch.cat([flat[t, :meta.valid_m(t), :hidden] for t in range(meta.num_row_tiles)])
    assert got.shape == (int(np.sum(lens)), hidden)
    assert torch.equal(got.view(torch.int16), want.contiguous().view(torch.int16))
