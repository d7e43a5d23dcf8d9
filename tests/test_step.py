"""A layer's call in one native step (ma_step): the same results, schedule and refusals as the calls
it stands for, for packed and paged keys; calls it does not take go the general way."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

from cases import CASES, make_inputs
from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.runtime import FusedFaOprojArWorkspace, FusedPrefillLayer
from megaattention_b200.runtime.workspace import StepMeta, claim_order
from oracle.chain_oracle import make_paged_kv

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include", "megaattn_b200.h")
FIELDS = ("cu_seqlens_q", "cu_seqlens_k", "cu_m_blocks", "batch_idx", "m_block")


def _cu(lens):
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


def _same_schedule(got, want):
    assert (got.num_batch, got.num_row_tiles, got.M_TILE) == (want.num_batch, want.num_row_tiles, 128)
    for f in FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        assert a.dtype == b.dtype and np.array_equal(a, b), f


def test_the_struct_is_the_headers(tmp_path):
    names = [(s, f) for s, t in (("ma_step_args", _cabi.StepArgs), ("ma_stage_tasks_args", _cabi.StageTasksArgs))
             for f, *_ in t._fields_]
    src = tmp_path / "l.c"
    src.write_text('#include <stdio.h>\n#include <stddef.h>\n#include "%s"\nint main(void) {\n' % HEADER
                   + "".join('printf("%%zu\\n", offsetof(%s, %s));\n' % n for n in names)
                   + 'printf("%zu %d\\n", sizeof(ma_step_args), MA_STEP_BLOCKS);return 0;}\n')
    subprocess.run(["gcc", "-std=c99", "-o", str(tmp_path / "l"), str(src)], check=True)
    out = subprocess.run([str(tmp_path / "l")], check=True, capture_output=True, text=True).stdout.split()
    types = {"ma_step_args": _cabi.StepArgs, "ma_stage_tasks_args": _cabi.StageTasksArgs}
    assert [int(x) for x in out] == ([getattr(types[s], f).offset for s, f in names]
                                     + [C.sizeof(_cabi.StepArgs), _cabi.STEP_BLOCKS])


@pytest.mark.parametrize("rows,width,first,step", [
    (1, 1, 0, 512), (1, 1, 1, 512), (12, 41, 7, 512), (3, 2001, 100, 8192), (1, 40000, 16383, 16384),
    (3, 1 << 29, 5, (1 << 24) + 1), (2, (1 << 31) - 1, 77, 1 << 25), (5, (1 << 28) + 3, (1 << 25) - 1, 1 << 25)])
def test_every_entry_of_a_table_is_somebodys(tmp_path, rows, width, first, step):
    """csrc/paged.cuh on the host: a thread's entries are every step-th of a group of rows, and the groups
    (of 2^30 entries or a row) cover the table."""
    (tmp_path / "cuda_runtime.h").write_text(
        "#include <algorithm>\nusing std::min; using std::max;\n#define __device__\n#define __forceinline__ inline\n")
    src = tmp_path / "t.cpp"
    src.write_text('#include <stdio.h>\n#include "%s"\nint main() { ma::for_each_entry(%d, %d, %du, %du, '
                   '[](int b, int j) { printf("%%d %%d\\n", b, j); }); }\n'
                   % (os.path.join(os.path.dirname(HEADER), "..", "megaattention_b200", "csrc", "paged.cuh"),
                      rows, width, first, step))
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-o", str(tmp_path / "t"), str(src)], check=True)
    got = [tuple(map(int, x.split())) for x in subprocess.run(
        [str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.splitlines()]
    group = max(1, (1 << 30) // width)
    want = [(b0 + i // width, i % width) for b0 in range(0, rows, group)
            for i in range(first, min(group, rows - b0) * width, step)]
    assert got == want


@pytest.mark.parametrize("q,k", [([3, 200, 128], [3, 900, 128]), ([1], [1])])
def test_the_schedule_is_made_when_looked_at(q, k):
    want = build_row_desc(q, seqlens_k=k)
    cu_q, lens = _cu(q), np.array(k, dtype=np.int32)
    for meta in (StepMeta(cu_q, lens, None, want.num_row_tiles), StepMeta(cu_q, None, _cu(k), want.num_row_tiles)):
        keep, keep_k = cu_q.copy(), lens.copy()
        cu_q[:], lens[:] = -5, -5                    # (the caller's again)
        _same_schedule(meta, want)
        cu_q[:], lens[:] = keep, keep_k


def _layer(name, paged):
    sq, H, hidden, qpk, sk, _ = CASES[name]
    sk = sq if sk is None else sk
    Q, K, V, W = make_inputs(name)
    kw, kv, pages = {}, (K, V), None
    if paged:
        pages = sum((s + 127) // 128 for s in sk) + 3
        Kc, Vc, table, lens = make_paged_kv(K, V, sk, num_pages=pages, shuffle=True, seed=5)
        kw = dict(paged=True, max_num_pages=pages, max_num_pages_per_seq=table.shape[1] + 2)
        kv = (Kc, Vc, table.cuda(), lens.cuda())
    R = sum((s + 127) // 128 for s in sq)
    ws = FusedFaOprojArWorkspace.create(None, R + 2, hidden, H, 128, q_per_kv=qpk, max_num_batch=len(sq) + 1,
                                        max_tot_k=sum(sk) + 64, device="cuda:0", **kw)
    ws.compile(w_fa=2, w_oproj=1, w_ar=0)
    layer = FusedPrefillLayer(ws, W)
    args = [Q.cuda(), kv[0].cuda(), kv[1].cuda(), torch.from_numpy(_cu(sq))]
    kwargs = dict(page_table=kv[2], cache_seqlens=kv[3]) if paged else dict(cu_seqlens_k=torch.from_numpy(_cu(sk)))
    return ws, layer, args, kwargs, build_row_desc(sq, seqlens_k=sk), pages


@pytest.mark.gpu
@pytest.mark.parametrize("paged", [False, True])
def test_a_step_is_what_the_calls_it_stands_for_are(paged):
    ws, layer, args, kwargs, want, pages = _layer("chunk_multiseq", paged)
    outs, metas, tables = [], [], []
    for native in (True, False, True):
        ws.can_step, saved = (ws.can_step if native else lambda *t: False), ws.can_step
        ws.csym.zero_()
        ws.meta_dev.zero_()
        out = layer(*args, **kwargs)
        ws.check_status()
        assert out.shape[0] == want.num_row_tiles and isinstance(layer.meta, StepMeta) == native
        outs.append((layer.output().clone(), ws.csym.clone()))
        tables.append(ws.meta_dev.clone())
        metas.append(layer.meta)
        ws.can_step = saved
    for o, m, t in zip(outs, metas, tables):
        assert torch.equal(o[0], outs[0][0]) and torch.equal(o[1], outs[0][1]) and torch.equal(t, tables[0])
        _same_schedule(m, want)
    # calls that are not for it: another current stream, a page table with columns apart
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert not ws.can_step()
        layer(*args, **kwargs)
    s.synchronize()
    ws.check_status()
    assert torch.equal(layer.output(), outs[0][0])
    if paged:
        t = kwargs["page_table"]
        apart = t.t().contiguous().t()
        wide = torch.full((t.shape[0], t.shape[1] + 5), -9, dtype=torch.int32, device="cuda")
        wide[:, 3:3 + t.shape[1]] = t
        for table, native in ((apart, t.shape[0] == 1 or t.shape[1] == 1), (wide[:, 3:3 + t.shape[1]], True)):
            layer(*args, page_table=table, cache_seqlens=kwargs["cache_seqlens"])
            ws.check_status()
            assert isinstance(layer.meta, StepMeta) == native and torch.equal(layer.output(), outs[0][0])


def _refused(args, kwargs, pages):
    """Page tables and key lengths that a step has to refuse."""
    table, lens = kwargs["page_table"], kwargs["cache_seqlens"]
    bad = []
    for page in (-1, pages):
        for at in ((0, 0), (-1, -1)):
            t = table.clone()
            t[at] = page
            bad.append((t, lens))
    for n in (0, -4, int(args[3][1]) - 1, table.shape[1] * 128 + 1):
        x = lens.clone()
        x[0] = n
        bad.append((table, x))
    return bad


@pytest.mark.gpu
def test_refusals_leave_the_last_step_in_place():
    ws, layer, args, kwargs, want, pages = _layer("chunk_multiseq", True)
    layer(*args, **kwargs)
    ws.check_status()
    ref = layer.output().clone()
    ws.csym.zero_()
    own = (ws.page_table, ws.cache_seqlens, ws.meta_dev)
    before = [t.clone() for t in own]
    for t, x in _refused(args, kwargs, pages):
        with pytest.raises(AssertionError):
            layer(*args, page_table=t, cache_seqlens=x)
        assert all(torch.equal(a, b) for a, b in zip(own, before))
    q = args[0]
    for other in ([q[:-1], *args[1:]], [q.float(), *args[1:]], [q, args[1].cpu(), *args[2:]],
                  [q, args[1][:, :, :, :64], *args[2:]]):
        with pytest.raises(AssertionError):
            layer(*other, **kwargs)
    torch.cuda.synchronize()
    assert not bool(ws.csym.any())                       # nothing was launched
    assert all(torch.equal(a, b) for a, b in zip(own, before))
    ws.launch()                                          # the plan still has all of the first step
    ws.check_status()
    assert torch.equal(ws.output(), ref)
    layer(*args, **kwargs)
    ws.check_status()
    assert torch.equal(layer.output(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("paged", [False, True])
def test_values_with_fewer_rows_than_keys_are_refused(paged, native):
    """K's count is what both are read by; more values than keys are left alone as before."""
    ws, layer, args, kwargs, want, pages = _layer("chunk_multiseq", paged)
    if not native:
        ws.can_step = lambda *t: False
    layer(*args, **kwargs)
    ws.check_status()
    ref = layer.output().clone()
    q, k, v, cu = args
    with pytest.raises(AssertionError):
        layer(q, k, v[:-1].clone(), cu, **kwargs)
    more = torch.cat((v, torch.full_like(v[:1], 7.0)))
    layer(q, k, more, cu, **kwargs)
    ws.check_status()
    assert torch.equal(layer.output(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("prime", [-(2 ** 40), -1, 0, 2, 2 ** 31, 2 ** 40])
def test_a_pinned_claim_order_of_any_size(prime):
    ws, layer, args, kwargs, want, _ = _layer("chunk_multiseq", False)
    ws.fa_prime_tiles = prime
    layer(*args, **kwargs)
    ws.check_status()
    assert isinstance(layer.meta, StepMeta)
    assert ws.fa_order[:want.num_row_tiles].tolist() == claim_order(want, prime).tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("paged", [False, True])
def test_launch_flags_that_are_refused_leave_the_plans_inputs(paged):
    """A workspace on its own buffers keeps them, and one that reads a caller's keeps those."""
    ws, layer, args, kwargs, want, pages = _layer("chunk_multiseq", paged)
    kv = dict(page_table=kwargs["page_table"], cache_seqlens=kwargs["cache_seqlens"]) if paged else {}
    ws.set_layer(want, *args[:3], layer.W_o, **kv)
    ws.launch()
    ws.check_status()
    ref, before = ws.output().clone(), ws.meta_dev.clone()
    others = [torch.zeros_like(t) for t in args[:3]] + args[3:]
    for first in (lambda: None, lambda: layer(*args, **kwargs)):
        first()
        bound = getattr(ws, "_bound", None)
        for flags in (_cabi.MA_FLAG_AR_ONLY, 1 << 20, _cabi.MA_FLAG_FA_ONLY | _cabi.MA_FLAG_OPROJ_ONLY):
            assert ws.can_step()
            with pytest.raises(RuntimeError):
                layer(*others, **kwargs, flags=flags)
        assert getattr(ws, "_bound", None) is bound and torch.equal(ws.meta_dev, before)
        ws.csym.zero_()
        ws.launch()
        ws.check_status()
        assert torch.equal(ws.output(), ref)
        ws.csym.zero_()
        ws.set_layer(want, *args[:3], layer.W_o, **kv)
        ws.launch()
        ws.check_status()
        assert torch.equal(ws.output(), ref)


@pytest.mark.gpu
def test_a_captured_launch_after_refusals():
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ws, layer, args, kwargs, want, pages = _layer("chunk_multiseq", True)
        layer(*args, **kwargs)
        ws.check_status()
        ref = layer.output().clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            ws.launch()
        for t, x in _refused(args, kwargs, pages):
            assert ws.can_step(t, x)
            with pytest.raises(AssertionError):
                layer(*args, page_table=t, cache_seqlens=x)
            ws.csym.zero_()
            graph.replay()
            ws.check_status()
            assert torch.equal(ws.output(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [1, 300, 2000, 40000])       # one block, a few, all of them
def test_a_table_of_any_width_is_copied_and_looked_through(width):
    ws, layer, args, kwargs, want, pages = _layer("chunk_gqa_q4", True)
    table, lens = kwargs["page_table"], kwargs["cache_seqlens"]
    more = torch.randint(0, pages, (table.shape[0], width), dtype=torch.int32, device="cuda")
    table = torch.cat((table, more), 1)
    _, H, hidden, qpk, _, _ = CASES["chunk_gqa_q4"]
    ws = FusedFaOprojArWorkspace.create(None, want.num_row_tiles, hidden, H, 128, q_per_kv=qpk, paged=True,
                                        max_num_pages=pages, max_num_pages_per_seq=table.shape[1] + 1,
                                        max_num_batch=want.num_batch, device="cuda:0").compile()
    big = FusedPrefillLayer(ws, layer.W_o)
    layer(*args, **kwargs)
    big(*args, page_table=table, cache_seqlens=lens)
    ws.check_status()
    assert isinstance(big.meta, StepMeta) and torch.equal(big.output(), layer.output())
    assert torch.equal(ws.page_table[:, :table.shape[1]], table) and not ws.page_table[:, table.shape[1]:].any()
    for at in ((0, 0), (table.shape[0] - 1, table.shape[1] - 1), (0, table.shape[1] // 2)):
        t = table.clone()
        t[at] = pages
        with pytest.raises(AssertionError):
            big(*args, page_table=t, cache_seqlens=lens)
