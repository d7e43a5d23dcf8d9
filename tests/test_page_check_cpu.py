"""What the page numbers of a paged call are checked by (runtime/prefill_layer.py): the table
itself below 16384 entries, its extremes from there on.  A page number goes into a TMA
coordinate, so both have to show one that is out of range wherever it stands."""
import numpy as np
import pytest
import torch

from megaattention_b200.runtime.prefill_layer import _lengths_and_pages


@pytest.mark.parametrize("width", [1, 5, 2047, 2048, 2049, 9000])       # 8 rows: 16384 is 2048 wide
@pytest.mark.parametrize("sliced", [False, True])
def test_lengths_and_the_range_of_the_pages(width, sliced):
    lens = torch.arange(3, 11, dtype=torch.int32)
    table = torch.randint(2, 90, (8, width + sliced), dtype=torch.int32)[:, int(sliced):]
    for at, page in (((0, 0), -1), ((7, width - 1), -1), ((0, 0), 100), ((7, width - 1), 100),
                     ((3, width // 2), 1)):
        t = table.clone() if not sliced else torch.cat((table[:, :1], table), 1)[:, 1:]
        t[at] = page
        got, pages = _lengths_and_pages(lens, t)
        assert got.dtype == np.int64 and got.tolist() == lens.tolist()
        assert int(pages.min()) == int(t.min()) and int(pages.max()) == int(t.max())
        assert page in (int(pages.min()), int(pages.max()))


def test_an_empty_table_is_left_to_the_caller():
    got, pages = _lengths_and_pages(torch.tensor([7], dtype=torch.int32), torch.zeros(1, 0, dtype=torch.int32))
    assert got.tolist() == [7] and pages is None
