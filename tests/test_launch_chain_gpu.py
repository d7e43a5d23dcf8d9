"""Kernels that start while the one before them is on its way out: a block's chain of calls queued
without a wait gives, bit for bit, what it gives with a wait after every call; and in a graph."""
import numpy as np
import pytest
import torch

from megaattention_b200 import _cabi
from megaattention_b200.metadata import build_row_desc
from megaattention_b200.runtime import FusedFaOprojArWorkspace, FusedPrefillLayer, residual_rmsnorm, rope_qk_

pytestmark = pytest.mark.gpu


def _upload_launches(ws, meta):
    """Of the metadata upload: up to 7680 words travel with each (csrc/meta_upload.cu)."""
    words = 2 * (meta.num_batch + 1) + 3 * meta.num_row_tiles + 6 + 4 + _cabi.TASK_WORDS * int(ws.tasks[0])
    return -(-words // 7680)


@pytest.mark.parametrize("q,uploads", [([64, 200], 1), ([128 * 40], 1), ([1] * 90, 1), ([1] * 700, 2)])
def test_a_chain_of_blocks(q, uploads):
    H, Hkv, hidden, n = 8, 2, 512, sum(q)
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev).to(torch.bfloat16)      # noqa: E731
    meta = build_row_desc(q)
    ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, hidden, H, 128, q_per_kv=H // Hkv,
                                        max_num_batch=len(q), device=dev).compile()
    layers = [FusedPrefillLayer(ws, rnd(H * 128, hidden) * 0.03) for _ in range(3)]
    mix = [rnd(hidden, H * 128) * 0.04 for _ in layers]
    kv = [(rnd(n, Hkv, 128), rnd(n, Hkv, 128)) for _ in layers]
    x0, weight = rnd(n, hidden), rnd(hidden)
    cu = np.concatenate([[0], np.cumsum(q)])

    def chain(wait):
        res = x0.clone()
        h, outs = res, []
        for layer, w, (k, v) in zip(layers, mix, kv):
            query, key = (h @ w).view(n, H, 128), k.clone()
            wait()
            rope_qk_(query, key, cu)
            wait()
            layer(query, key, v, cu)
            wait()
            h, res = residual_rmsnorm(ws, res, weight, 1e-6)
            wait()
            outs += [query, key, layer.output(), h, res]
            wait()
        return outs

    want = chain(torch.cuda.synchronize)
    for _ in range(5):
        got = chain(lambda: None)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    ws.check_status()
    assert _upload_launches(ws, meta) == uploads


@pytest.mark.parametrize("q,uploads", [([300, 40], 1), ([1] * 1300, 3)])
def test_launches_in_a_graph(q, uploads):
    dev = torch.device("cuda:0")
    meta = build_row_desc(q)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ws = FusedFaOprojArWorkspace.create(None, meta.num_row_tiles, 256, 4, 128, q_per_kv=4, device=dev).compile()
        ws.Q.normal_(); ws.K.normal_(); ws.V.normal_(); ws.W_o.normal_(std=0.04)
        ws.set_meta(meta)
        ws.launch()
        want = ws.output()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            ws.set_meta(meta)
            ws.launch()
            got = ws.output()
            ws.launch()
            again = ws.output()
        for _ in range(3):
            ws.csym.zero_(); got.zero_(); again.zero_()
            graph.replay()
            s.synchronize()
            assert torch.equal(got, want) and torch.equal(again, want)
        ws.check_status()
        assert _upload_launches(ws, meta) == uploads
