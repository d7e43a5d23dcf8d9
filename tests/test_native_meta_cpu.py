"""The native host metadata (csrc/meta.cpp) against the numpy statement of the same arithmetic
(metadata/row_desc.py, runtime/workspace.claim_order): random batches, every claim order, every
rank of several sizes, and the batches that both refuse."""
import ctypes as C

import numpy as np
import pytest

from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.metadata.launch_heuristic import fa_prime_tiles_b200
from megaattention_b200.metadata.row_desc import active_counts
from megaattention_b200.runtime.workspace import claim_order, native_row_desc


def _cu(lens):
    return np.concatenate([[0], np.cumsum(lens)])


def _batches():
    rng = np.random.RandomState(5)
    yield [1], [1]
    yield [128], [128]
    yield [129, 128, 127, 1], [4000, 128, 300, 1]
    for _ in range(60):
        n = rng.randint(1, 40)
        q = rng.randint(1, 900, size=n)
        yield q.tolist(), (q + rng.randint(0, 3000, size=n) * rng.randint(0, 2)).tolist()


def test_row_desc_and_staging_match_numpy():
    rng = np.random.RandomState(6)
    for q, k in _batches():
        want = build_row_desc(q, seqlens_k=k)
        got = native_row_desc(_cu(q), _cu(k), 1 << 20)
        R, nb = want.num_row_tiles, want.num_batch
        assert (got.num_row_tiles, got.num_batch, got.M_TILE) == (R, nb, 128)
        for f in ("cu_seqlens_q", "cu_seqlens_k", "cu_m_blocks", "batch_idx", "m_block"):
            a, b = getattr(got, f), getattr(want, f)
            assert a.dtype == b.dtype == np.int32 and np.array_equal(a, b), f
        hidden, H, nsg = int(rng.choice([128, 1000, 4096])), int(rng.choice([1, 8])), int(rng.choice([1, 8]))
        tp = int(rng.choice([1, 2, 8]))
        rank = int(rng.randint(0, tp))
        offs = np.cumsum([0, nb + 1, nb + 1, R, R, R])
        for prime in (None, 0, -1, 1, 3, R, R + 7):
            buf = np.full(int(offs[-1]) + 8, -9, dtype=np.int32)
            a = _cabi.StageMetaArgs(
                got.cu_seqlens_q.ctypes.data, got.cu_seqlens_k.ctypes.data, got.batch_idx.ctypes.data,
                got.m_block.ctypes.data, buf.ctypes.data, nb, R, hidden, H, nsg, tp, rank,
                int(prime is None), prime or 0, *map(int, offs), 0)
            assert _cabi.lib.ma_stage_meta(C.byref(a)) == _cabi.MA_OK
            p = fa_prime_tiles_b200(want, hidden, tp, H) if prime is None else prime
            parts = (want.cu_seqlens_q, want.cu_seqlens_k, want.batch_idx, want.m_block,
                     claim_order(want, p), active_counts(R, H, nsg, tp, rank))
            assert np.array_equal(buf[:-2], np.concatenate(parts)) and (buf[-2:] == -9).all()


@pytest.mark.parametrize("q,k", [([3, 0], [3, 4]), ([5], [4]), ([-1, 4], [2, 4])])
def test_refused_batches_stay_refused(q, k):
    with pytest.raises(AssertionError):
        build_row_desc(q, seqlens_k=k)
    with pytest.raises(AssertionError):
        native_row_desc(_cu(q), _cu(k), 100)


def test_more_tiles_than_the_bound_is_refused():
    assert native_row_desc([0, 257], [0, 257], 3).num_row_tiles == 3
    with pytest.raises(AssertionError):
        native_row_desc([0, 257], [0, 257], 2)


def test_key_lengths_may_sum_past_int32():
    """Paged sequences share pages, so a batch's key lengths may sum past 2^31 - 1; the numpy
    statement narrows the sum and goes on, and so does the native one, with the true lengths in
    the claim order."""
    big = 1 << 30
    q, k = [1, 300, 1, 200], [big, big + 256, big - 128, 250]
    want, got = build_row_desc(q, seqlens_k=k), native_row_desc(_cu(q), _cu(k), 100)
    for f in ("cu_seqlens_q", "cu_seqlens_k", "cu_m_blocks", "batch_idx", "m_block"):
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
    R, nb = got.num_row_tiles, got.num_batch
    offs = np.cumsum([0, nb + 1, nb + 1, R, R, R])
    buf = np.zeros(int(offs[-1]) + 6, dtype=np.int32)
    for meta in (got, want):
        a = _cabi.StageMetaArgs(
            meta.cu_seqlens_q.ctypes.data, meta.cu_seqlens_k.ctypes.data, meta.batch_idx.ctypes.data,
            meta.m_block.ctypes.data, buf.ctypes.data, nb, R, 4096, 8, 8, 1, 0, 0, 0, *map(int, offs), 0)
        assert _cabi.lib.ma_stage_meta(C.byref(a)) == _cabi.MA_OK
        # key blocks beyond 2^23: 0 | 1, 2, 2 | -1; the last sequence has two a tile
        assert buf[offs[4]:offs[5]].tolist() == [2, 3, 1, 0, 4, 5, 6]
    with pytest.raises(AssertionError):
        native_row_desc(_cu([1]), _cu([1 << 31]), 100)


@pytest.mark.parametrize("hidden,interleaved", [(257, True), (256, False), (384, True), (1, False)])
def test_the_claim_order_switches_where_the_rule_does(hidden, interleaved):
    """fa_prime_tiles_b200 and ma_stage_meta each have the switch point; a batch whose work ratio
    is exactly 2 (one sequence of three row tiles, two column tiles: 2 * 6 / 6) and its
    neighbours take the same side in both."""
    meta = build_row_desc([384])
    p = fa_prime_tiles_b200(meta, hidden, 1, 8)
    assert (p < 0) == interleaved
    R, nb = 3, 1
    offs = np.cumsum([0, nb + 1, nb + 1, R, R, R])
    buf = np.zeros(int(offs[-1]) + 6, dtype=np.int32)
    a = _cabi.StageMetaArgs(
        meta.cu_seqlens_q.ctypes.data, meta.cu_seqlens_k.ctypes.data, meta.batch_idx.ctypes.data,
        meta.m_block.ctypes.data, buf.ctypes.data, nb, R, hidden, 8, 1, 1, 0, 1, 0, *map(int, offs), 0)
    assert _cabi.lib.ma_stage_meta(C.byref(a)) == _cabi.MA_OK
    assert buf[offs[4]:offs[5]].tolist() == claim_order(meta, p).tolist()
    assert claim_order(meta, p).tolist() == ([2, 0, 1] if interleaved else [2, 1, 0])
