"""The O_proj task shapes of a single rank (row tiles x column tiles: 2 x 2, 1 x 2, 1 x 1,
chosen by the number of 2 x 2 tasks per CTA) against the oracle: odd numbers of row tiles and
of column tiles, a partial row tile in either half of a pair, a hidden size that ends inside
a tile.  The CTA count picks the shape: with t 2 x 2 tasks, n CTAs, 2 x 2 from t >= 3 n, two
column tiles from 4 t >= 5 n."""
import pytest

from test_fused_single_gpu import CASES, check, run_case

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
