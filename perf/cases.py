"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is one layer of prefill for one batch of sequences on one GPU (one tensor-parallel
rank's share of the heads), through the public entry points, in one of four forms:

``layer``      ``FusedPrefillLayer`` on packed Q/K/V: a complete prompt, or a chunk whose keys
               are packed with it.
``paged``      ``FusedPrefillLayer`` on a paged KV cache (128-token pages, shuffled page table
               and lengths on the device): chunked prefill and prefix-cached prompts.
``step``       the layer between its neighbours, as a transformer block runs it:
               ``rope_qk_`` -> ``FusedPrefillLayer`` -> ``residual_rmsnorm`` (in place).
``workspace``  the plain workspace interface: ``set_layer`` (copies the inputs in), ``launch``,
               ``output`` (de-tiled result).

Sizes are this repository's benchmark configurations (``megaattention_b200/workloads.py``), a
shape of its calibration sweep, and generic serving shapes.  Inputs are N(0, 1) bf16 with
weights of std ``fan_in ** -0.5``, as in those benchmarks.
"""
import math

import numpy as np
import torch

from megaattention_b200.metadata import build_row_desc, choose_launch_config
from megaattention_b200.runtime import (
    FusedFaOprojArWorkspace, FusedPrefillLayer, residual_rmsnorm, rope_qk_)
from megaattention_b200.runtime.rope import default_inv_freq, rope_meta

D = 128
PAGE = 128


def _case(name, form, q, heads, kv_heads, hidden, k=None):
    return {"name": name, "form": form, "q": ",".join(map(str, q)),
            "k": ",".join(map(str, q if k is None else k)),
            "heads": heads, "kv_heads": kv_heads, "hidden": hidden}


_SMALL = [6800, 2900, 1700, 1100, 600, 300]
_SWEEP = [7500, 4100, 3300, 2600, 2000, 1500, 1000, 600]
# a prefix-cached batch: short new turns behind conversations of a few thousand tokens
_TURNS_Q = [17, 256, 45, 130, 300, 64, 1, 97, 211, 33, 150, 80]
_TURNS_K = [2065, 3300, 801, 1154, 4396, 640, 1537, 5217, 1235, 2800, 150, 3152]


def listed():
    return [
        # a few short prompts on a small model: latency of the whole call
        _case("layer_short", "layer", [64, 200, 256], 8, 1, 1024),
        # new turns of a dozen prefix-cached conversations in one step
        _case("paged_turns", "paged", _TURNS_Q, 8, 1, 4096, _TURNS_K),
        # one 2000-token chunk at the end of a 16k context (chunked prefill)
        _case("paged_chunk", "paged", [2000], 8, 1, 4096, [15871]),
        # four equal prompts, a whole block's neighbouring ops around the layer
        _case("step_uniform", "step", [1024] * 4, 16, 2, 2048),
        # ordinary ragged batch, one rank of an 8-way split model
        _case("layer_ragged", "layer", _SMALL, 8, 1, 4096),
        # the same batch without grouped heads
        _case("layer_mha", "layer", _SMALL, 8, 8, 4096),
        # the same batch through the copying interface, result de-tiled
        _case("workspace_ragged", "workspace", _SMALL, 8, 1, 4096),
        # chunked prefill of the ragged batch: three quarters of the keys are cached
        _case("paged_prefix", "paged", _SMALL, 8, 1, 4096, [4 * n for n in _SMALL]),
        # one long prompt: the attention dominates
        _case("layer_long", "layer", [16384], 8, 1, 2048),
        # larger batch, one rank of a 4-way split model, with the neighbouring ops
        _case("step_sweep", "step", _SWEEP, 16, 2, 4096),
        # wide model: the projection dominates
        _case("layer_wide", "layer", _SWEEP, 16, 1, 16384),
        # the whole 64-head model on one GPU
        _case("layer_whole", "layer", _SWEEP, 64, 8, 4096),
    ]


def _lens(case):
    return [int(x) for x in case["q"].split(",")], [int(x) for x in case["k"].split(",")]


def work(case):
    """Un-padded causal attention and projection FLOPs; each input read and each output
    written once."""
    q, k = _lens(case)
    H, Hkv, hid = case["heads"], case["kv_heads"], case["hidden"]
    tq, tk = sum(q), sum(k)
    flops = sum(4.0 * D * H * (a * (b - a) + a * (a + 1) / 2) for a, b in zip(q, k))
    flops += 2.0 * tq * H * D * hid
    nbytes = 2.0 * (tq * H * D + 2 * tk * Hkv * D + H * D * hid + tq * hid)
    if case["form"] == "step":
        # rotated q and k written back; residual read and written, normalised output written
        nbytes += 2.0 * (tq * H * D + tq * Hkv * D + 3 * tq * hid)
    return {"bytes": nbytes, "flops": flops}


def draw(rng):
    """One more case of these ranges: 200 to 24000 new tokens in 1 to 24 sequences of uneven
    lengths, the head groupings and widths that models have, never more work than
    ``layer_whole``."""
    most = work(listed()[-1])
    while True:
        form = rng.choice(["layer", "layer", "paged", "paged", "step", "workspace"])
        heads, kv = rng.choice([(8, 1), (8, 1), (8, 8), (16, 2), (16, 1), (4, 1), (7, 1),
                                (6, 2), (12, 12), (32, 4), (64, 8)])
        hidden = 8 * round(math.exp(rng.uniform(math.log(512), math.log(16384))) / 8)
        tokens = math.exp(rng.uniform(math.log(200), math.log(24000)))
        n = round(math.exp(rng.uniform(0.0, math.log(24))))
        share = [rng.uniform(0.2, 1.0) ** 2 for _ in range(n)]
        q = [max(1, round(tokens * s / sum(share))) for s in share]
        k = list(q)
        if form == "paged" or (form == "layer" and rng.random() < 0.25):
            longest = math.exp(rng.uniform(math.log(128), math.log(16000)))
            k = [a + round(longest * rng.random()) for a in q]
        c = _case("drawn", form, q, heads, kv, hidden, k)
        del c["name"]
        w = work(c)
        if w["flops"] <= most["flops"] and w["bytes"] <= 2 * most["bytes"] and sum(k) <= 200000:
            return c


def tolerance(case):
    """The path rounds P, the attention output and the result to bf16: against the same chain
    in fp32 it is off by 2.5e-3 to 3e-3 in the 2-norm and by up to 2e-2 at single elements
    (small cases; the 2e-2 grows slowly with the number of elements).  Four times that."""
    return {"rel": 1e-2, "max": 0.1}


def _inputs(case, seed):
    """The case's tensors, from the seed alone."""
    q, k = _lens(case)
    H, Hkv, hid = case["heads"], case["kv_heads"], case["hidden"]
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))

    def randn(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device=dev, dtype=torch.bfloat16) * std).contiguous()

    tq, tk = sum(q), sum(k)
    t = {"W_o": randn(H * D, hid, std=(H * D) ** -0.5), "q": randn(tq, H, D)}
    if case["form"] == "paged":
        need = [-(-n // PAGE) for n in k]
        pages = sum(need) + 8
        perm = np.random.RandomState(int(seed) % (1 << 31)).permutation(pages).astype(np.int32)
        table = np.zeros((len(k), max(need)), dtype=np.int32)
        at = 0
        for i, n in enumerate(need):
            table[i, :n] = perm[at:at + n]
            at += n
        t["k"], t["v"] = randn(pages * PAGE, Hkv, D), randn(pages * PAGE, Hkv, D)
        t["pages"] = pages
        t["page_table"] = torch.from_numpy(table).to(dev)
        t["cache_seqlens"] = torch.tensor(k, dtype=torch.int32, device=dev)
    else:
        t["k"], t["v"] = randn(tk, Hkv, D), randn(tk, Hkv, D)
    if case["form"] == "step":
        t["residual"] = randn(tq, hid)
        t["weight"] = (1.0 + 0.1 * randn(hid)).contiguous()
    return t


def prepare(case, seed):
    q, k = _lens(case)
    H, Hkv, hid, form = case["heads"], case["kv_heads"], case["hidden"], case["form"]
    dev = torch.device("cuda:0")
    meta = build_row_desc(q, seqlens_k=k)
    cfg = choose_launch_config(meta, hid, 1)
    s = {"form": form, "meta": meta, **_inputs(case, seed)}
    kw = {}
    if form == "paged":
        kw = dict(paged=True, max_num_pages=s["pages"],
                  max_num_pages_per_seq=s["page_table"].shape[1])
    ws = FusedFaOprojArWorkspace.create(
        None, meta.num_row_tiles, hid, H, D, super_group_n_tiles=cfg.sg, q_per_kv=H // Hkv,
        max_num_batch=meta.num_batch, max_tot_k=sum(k), device=dev, **kw)
    ws.compile(w_fa=cfg.w_fa, w_oproj=cfg.w_oproj, w_ar=cfg.w_ar)
    s["ws"] = ws
    s["cu_q"] = torch.from_numpy(meta.cu_seqlens_q)
    s["cu_k"] = torch.from_numpy(meta.cu_seqlens_k)
    if form != "workspace":
        s["layer"] = FusedPrefillLayer(ws, s["W_o"])
    if form == "step":
        s["rope"] = rope_meta(meta.cu_seqlens_q, meta.cu_seqlens_k, dev)
        s["inv_freq"] = default_inv_freq(10000.0, dev)
    return s


def _rotated(x, pos):
    """Rotate-half RoPE of ``x [n, heads, 128]`` (float64) at positions ``pos [n]``."""
    freq = 10000.0 ** (-torch.arange(0, D, 2, dtype=torch.float64, device=x.device) / D)
    ang = pos.double()[:, None] * freq
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def exact(case, seed):
    """What ``run`` returns, in float64 from the definition."""
    lens_q, lens_k = _lens(case)
    H, Hkv, hid, form = case["heads"], case["kv_heads"], case["hidden"], case["form"]
    if work(case)["flops"] > 1.5e12:          # minutes in float64
        return None
    t = _inputs(case, seed)
    dev = t["q"].device
    q, k, v = t["q"].double(), t["k"].double(), t["v"].double()
    W = t["W_o"].double()
    tiles = sum(-(-n // 128) for n in lens_q)
    out = torch.zeros(tiles * 128, -(-hid // 128) * 128, dtype=torch.float64, device=dev)
    packed = torch.empty(sum(lens_q), hid, dtype=torch.float64, device=dev)
    q0 = k0 = row = 0
    for i, (lq, lk) in enumerate(zip(lens_q, lens_k)):
        if form == "paged":
            idx = (t["page_table"][i].long()[:, None] * PAGE
                   + torch.arange(PAGE, device=dev)).reshape(-1)[:lk]
        else:
            idx = torch.arange(k0, k0 + lk, device=dev)
        if form == "step":
            pos = torch.arange(lk - lq, lk, device=dev)
            q[q0:q0 + lq] = _rotated(q[q0:q0 + lq], pos)
            k[idx[lk - lq:]] = _rotated(k[idx[lk - lq:]], pos)
        ks, vs = k[idx], v[idx]
        attn = torch.empty(lq, H, D, dtype=torch.float64, device=dev)
        for h in range(H):
            for a in range(0, lq, 1024):
                e = min(lq, a + 1024)
                n = lk - lq + e                # keys the last of these rows may see
                sc = q[q0 + a:q0 + e, h] @ ks[:n, h * Hkv // H].T * D ** -0.5
                seen = torch.arange(lk - lq + a, n, device=dev)[:, None]
                sc.masked_fill_(torch.arange(n, device=dev) > seen, -math.inf)
                attn[a:e, h] = torch.softmax(sc, dim=-1) @ vs[:n, h * Hkv // H]
        packed[q0:q0 + lq] = attn.view(lq, H * D) @ W
        out[row:row + lq, :hid] = packed[q0:q0 + lq]
        q0, k0, row = q0 + lq, k0 + lk, row + -(-lq // 128) * 128
    if form == "workspace":
        return packed
    out = out.view(tiles, 128, -1, 128)
    if form != "step":
        return out
    res = t["residual"].double() + packed
    normed = res * torch.rsqrt(res.square().mean(-1, keepdim=True) + 1e-6) * t["weight"].double()
    return {"attn": out, "normed": normed, "residual": res, "q": q, "k": k}


def run(s):
    form = s["form"]
    if form == "workspace":
        ws = s["ws"]
        ws.set_layer(s["meta"], s["q"], s["k"], s["v"], s["W_o"])
        ws.launch()
        return ws.output()
    if form == "paged":
        return s["layer"](s["q"], s["k"], s["v"], s["cu_q"], page_table=s["page_table"],
                          cache_seqlens=s["cache_seqlens"])
    if form == "layer":
        return s["layer"](s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"])
    rope_qk_(s["q"], s["k"], meta=s["rope"], inv_freq=s["inv_freq"])
    attn = s["layer"](s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"])
    normed, residual = residual_rmsnorm(s["ws"], s["residual"], s["weight"], 1e-6, inplace=True)
    return {"attn": attn, "normed": normed, "residual": residual, "q": s["q"], "k": s["k"]}
