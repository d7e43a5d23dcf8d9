"""A launch does not need all of its CTAs at once: what another stream's kernel keeps from an SM
is done by the CTAs that run, within their wait limit, and a late CTA finds the work done.
(The claim rule itself, with one CTA late, is in test_protocol_model_cpu.py.)"""
import time

import pytest
import torch

from cases import _randn
from oracle.chain_oracle import err_beyond_rounding, full_chain_oracle

pytestmark = pytest.mark.gpu


# more attention tasks (160, two heads each) than the GPU has SMs
SQ, H, HIDDEN, QPK = [130] * 20, 8, 256, 8


def _inputs():
    n = sum(SQ)
    return (_randn((n, H, 128), 4100), _randn((n, H // QPK, 128), 4101),
            _randn((n, H // QPK, 128), 4102), _randn((H * 128, HIDDEN), 4103, float(H * 128) ** -0.5))


def _workspace(sq, hidden, stream, **compile_args):
    from megaattention_b200.metadata import build_row_desc
    from megaattention_b200.runtime import FusedFaOprojArWorkspace
    meta = build_row_desc(sq)
    with torch.cuda.stream(stream):
        ws = FusedFaOprojArWorkspace.create(
            None, meta.num_row_tiles, hidden, H, 128, q_per_kv=QPK,
            max_tot_k=int(meta.cu_seqlens_k[-1]), device="cuda:0")
        ws.compile(w_fa=2, w_oproj=1, w_ar=0, **compile_args)
    return ws, meta


def test_launch_beside_a_kernel_that_holds_some_sms():
    """Four CTAs of a long launch hold four SMs for several wait limits of a second, full-grid
    launch on another stream."""
    limit_ms, n = 8, 24576
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    long_ws, long_meta = _workspace([n], 128, s1, num_ctas=4)
    long_ws.Q.normal_(); long_ws.K.normal_(); long_ws.V.normal_()
    long_ws.set_meta(long_meta)
    Q, K, V, W = _inputs()
    ws, meta = _workspace(SQ, HIDDEN, s2, wait_limit_ms=limit_ms)
    ws.set_layer(meta, Q.cuda(), K.cuda(), V.cuda(), W.cuda())
    torch.cuda.synchronize()
    t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    t0.record(s1)
    long_ws.launch()
    t1.record(s1)
    time.sleep(0.002)
    ws.launch()
    torch.cuda.synchronize()
    assert t0.elapsed_time(t1) > 3 * limit_ms          # the other launch was in the way long enough
    ws.check_status()
    long_ws.check_status()
    _, Yp, _ = full_chain_oracle(Q, K, V, W, SQ)
    assert err_beyond_rounding(ws.output(meta).cpu(), Yp) <= 2e-3
    assert ws.ctrl.cpu().tolist() == [0] * 8 == long_ws.ctrl.cpu().tolist()


def test_full_grid_launches_on_two_streams():
    """Two workspaces launch again and again on two streams that nothing orders: each launch
    gets the SMs that the other leaves."""
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    Q, K, V, W = _inputs()
    _, Yp, _ = full_chain_oracle(Q, K, V, W, SQ)
    pairs = [_workspace(SQ, HIDDEN, s, wait_limit_ms=500) for s in streams]
    for ws, meta in pairs:
        ws.set_layer(meta, Q.cuda(), K.cuda(), V.cuda(), W.cuda())
    torch.cuda.synchronize()
    for _ in range(40):
        for ws, _m in pairs:
            ws.launch()
    torch.cuda.synchronize()
    for ws, meta in pairs:
        ws.check_status()
        assert err_beyond_rounding(ws.output(meta).cpu(), Yp) <= 2e-3
        assert ws.ctrl.cpu().tolist() == [0] * 8
