"""Long-lived workspace of the fused FlashAttention -> O_proj -> AllReduce kernel.

Same surface as the reference's ``FusedFaOprojArWorkspace``
(``src/mega_attention/runtime/workspace.py``): ``create`` (:46-150) allocates every buffer
once at a bucket capacity and, with ``tp_size > 1``, rendezvous-es the symmetric ones;
``compile`` (:174-194) fixes the launch configuration; ``set_layer`` (:197-235) fills the
active prefixes and the six active counts; ``launch`` (:237-240) runs one layer with no
host-side reset in between; ``debug_zero_all`` (:243-248) is for fault localisation only.

Differences a caller can observe:

* nothing is JIT-compiled: ``compile`` builds a plan through the C ABI
  (``ma_plan_create``) and the role weights / CTA count are launch arguments;
* ``set_layer`` validates *every* capacity before copying anything;
* device-side waits are bounded: ``check_status`` raises ``RuntimeError`` when one gave up;
* role weights and CTA count can change per ``compile`` without any rebuild.

torch is used for device memory, streams and (tp > 1) symmetric-memory bootstrap only.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import functools

import numpy as np
import torch

from .. import _cabi
from ..metadata.launch_heuristic import launch_flags_b200
from ..metadata.row_desc import RowDescMeta, oproj_task_counts

NUM_CTRL = 8
NUM_SYNC = 3
NUM_STATUS = 8
SPLIT_HEADS = 640        # (two waves of tasks of two heads, and a little)
MAX_PARTS = 16           # of one row tile, as in csrc/kparams.h


def claim_order(meta, prime: int = 0) -> np.ndarray:
    """Row tiles sorted by the number of 128-key blocks their attention task visits,
    longest first (stable), so the biggest tasks are claimed first and the tail of the
    launch is filled with small ones.  Same on every rank.

    ``prime`` > 0 moves that many of the shortest row tiles to the front: their attention
    finishes within microseconds, so O_proj and AllReduce work exists almost from the start
    of the launch instead of only after the first long attention task (tens of
    microseconds) — worth it when the launch is bound by the AllReduce.  ``prime`` < 0
    interleaves long and short row tiles instead (see below).

    A launch's order is computed natively (``csrc/meta.cpp``); this is the statement of it that
    the tests hold that to."""
    M = meta.M_TILE
    b = meta.batch_idx.astype(np.int64)
    lq = np.diff(meta.cu_seqlens_q.astype(np.int64))[b]
    lk = np.diff(meta.cu_seqlens_k.astype(np.int64))[b]
    last_row = (meta.m_block.astype(np.int64) + 1) * M + (lk - lq)
    nblk = np.minimum(-(-lk // M), -(-last_row // M))
    order = np.argsort(-nblk, kind="stable").astype(np.int32)
    if prime < 0:
        # interleaved: longest, shortest, second longest, second shortest, ...  Row tiles
        # then finish at an even rate from the start of the launch (steady O_proj and
        # AllReduce work) while the long tasks still start early; the last tasks claimed are
        # of middling length.
        out = np.empty_like(order)
        half = (order.size + 1) // 2
        out[0::2] = order[:half]
        out[1::2] = order[half:][::-1]
        return out
    prime = int(min(prime, order.size))
    if prime:
        order = np.concatenate([order[order.size - prime:][::-1], order[:order.size - prime]])
    return order


def native_row_desc(cu_q, cu_k, max_row_tiles: int) -> RowDescMeta:
    """``build_row_desc`` from cumulative lengths (int64 arrays), natively: the same object
    and the same refusals, a tenth of the host time.  ``max_row_tiles`` bounds the schedule."""
    cu_q = np.ascontiguousarray(cu_q, dtype=np.int64)
    cu_k = np.ascontiguousarray(cu_k, dtype=np.int64)
    nb = cu_q.size - 1
    assert nb > 0 and cu_k.size == nb + 1
    cap = int(max(0, min(max_row_tiles, int(cu_q[nb]) // 128 + nb)))
    buf = np.empty(3 * (nb + 1) + 2 * cap, dtype=np.int32)
    o_q, o_k, o_m = buf[:nb + 1], buf[nb + 1:2 * nb + 2], buf[2 * nb + 2:3 * nb + 3]
    base = buf.ctypes.data
    at = base + 12 * (nb + 1)
    n = _cabi.lib.ma_row_desc(cu_q.ctypes.data, cu_k.ctypes.data, nb, cap, base, base + 4 * (nb + 1),
                              base + 8 * (nb + 1), at, at + 4 * cap)
    assert n != _cabi.MA_ERR_INVALID, "0 < q_len <= k_len per sequence"
    assert n > 0, "more row tiles than the workspace was created for"
    at = 3 * (nb + 1)
    return RowDescMeta(num_batch=nb, M_TILE=128, cu_seqlens_q=o_q, cu_seqlens_k=o_k,
                       num_row_tiles=n, cu_m_blocks=o_m, batch_idx=buf[at:at + n],
                       m_block=buf[at + cap:at + cap + n])


class StepMeta(RowDescMeta):
    """The schedule of a step that was queued natively: its arrays are made when somebody looks."""

    def __init__(self, cu_q, lens_k, cu_k, num_row_tiles):
        self.num_batch, self.M_TILE, self.num_row_tiles = cu_q.size - 1, 128, num_row_tiles
        # (copies: the caller's arrays and the lengths' staging are their owners' again)
        self._cu_q = cu_q.copy()
        self._lens_k = None if lens_k is None else lens_k.copy()
        self._cu_k = self._cu_q if cu_k is cu_q else (None if cu_k is None else cu_k.copy())

    @functools.cached_property
    def _all(self):
        cu_k = self._cu_k
        if cu_k is None:
            cu_k = np.zeros(self.num_batch + 1, dtype=np.int64)
            np.cumsum(self._lens_k, out=cu_k[1:])
        return native_row_desc(self._cu_q, cu_k, self.num_row_tiles)

    @functools.cached_property
    def cu_seqlens_q(self):
        return self._cu_q.astype(np.int32)

    cu_seqlens_k = functools.cached_property(lambda self: self._all.cu_seqlens_k)
    cu_m_blocks = functools.cached_property(lambda self: self._all.cu_m_blocks)
    batch_idx = functools.cached_property(lambda self: self._all.batch_idx)
    m_block = functools.cached_property(lambda self: self._all.m_block)


class FusedFaOprojArWorkspace:
    def __init__(self, **kw):
        self.__dict__.update(kw)
        self._plan = None
        self._lib = _cabi.lib
        self._split_ctas = 0           # (set by compile: before it nothing is split)
        self._step_args = None
        self._args = None
        self._meta = None
        # Launch flags applied by launch() (OR of _cabi.MA_FLAG_*) and attention claim order
        # (see claim_order).  None = chosen for the batch at hand by the calibrated rules,
        # launch_flags_b200 / fa_prime_tiles_b200; an int pins the setting.
        self.default_flags = None
        self.fa_prime_tiles = None
        self._auto_flags = 0
        self.ar_p2p = True       # tp_size == 2: AllReduce through peer loads instead of multimem

    # ------------------------------------------------------------------ create
    @classmethod
    def create(cls, group_name, max_num_row_tiles, hidden, H_local, D,
               tp_size=1, rank=0, N_TILE=128, super_group_n_tiles=4, q_per_kv=1,
               max_num_batch=None, max_tot_k=None, dtype=torch.bfloat16, device=None,
               paged=False, page_size=128, max_num_pages=None,
               max_num_pages_per_seq=None, key_splits=True):
        """``key_splits=False`` leaves out the room for parts of long attention tasks (up to 42 MB,
        ``parts``): batches of few long sequences then run their row tiles whole."""
        assert dtype == torch.bfloat16 and D == 128 and N_TILE == 128
        assert H_local % q_per_kv == 0
        assert 1 <= super_group_n_tiles <= 4, "a super-group is at most 512 TMEM columns"
        dev = torch.device(device if device is not None
                           else f"cuda:{torch.cuda.current_device()}")
        H_kv = H_local // q_per_kv
        K_local = H_local * D
        if max_num_batch is None:
            max_num_batch = max_num_row_tiles
        num_out, nsg, max_total = oproj_task_counts(
            max_num_row_tiles, hidden, N_TILE, super_group_n_tiles)
        hidden_pad = num_out * N_TILE
        tot_cap = max_num_row_tiles * 128
        if max_tot_k is None:
            max_tot_k = tot_cap
        # paged KV: K/V live in [num_pages, 128, H_kv, D] caches addressed through a page
        # table; one page is exactly one 128-key block (workspace.py:67-74 of the reference)
        if paged:
            assert page_size == N_TILE == 128, (page_size, N_TILE)
            if max_num_pages is None:
                max_num_pages = (max_tot_k + 127) // 128
            if max_num_pages_per_seq is None:
                max_num_pages_per_seq = (max_tot_k + 127) // 128
        max_owner_slots = (max_total + tp_size - 1) // tp_size
        max_owner_words = (max_owner_slots + 63) // 64

        def zeros(shape, dt):
            return torch.zeros(shape, dtype=dt, device=dev)

        handles = None
        if tp_size > 1:
            import torch.distributed as dist
            import torch.distributed._symmetric_memory as symm_mem

            def sym(shape, dt):
                t = symm_mem.empty(*shape, device=dev, dtype=dt)
                t.zero_()
                return t, symm_mem.rendezvous(t, group_name)

            csym, hC = sym((max_num_row_tiles, 128, num_out, N_TILE), dtype)
            assert hC.has_multicast_support, "NVLS multicast is required for tp_size > 1"
            rco, hRC = sym((max_owner_slots,), torch.uint32)
            rbits, hRB = sym((max_owner_words,), torch.int64)
            nvl, hN = sym((2,), torch.int32)
            csym_mc_ptr = int(hC.multicast_ptr)
            rc_ptrs = [int(hRC.buffer_ptrs[r]) for r in range(tp_size)]
            rb_ptrs = [int(hRB.buffer_ptrs[r]) for r in range(tp_size)]
            nvl_peer_ptrs = [int(hN.buffer_ptrs[r]) for r in range(tp_size)]
            csym_peer_ptrs = [int(hC.buffer_ptrs[r]) for r in range(tp_size)]
            handles = (hC, hRC, hRB, hN)
        else:
            csym = zeros((max_num_row_tiles, 128, num_out, N_TILE), dtype)
            rco = zeros(max_owner_slots, torch.uint32)
            rbits = zeros(max_owner_words, torch.int64)
            nvl = zeros(2, torch.int32)
            csym_mc_ptr = 0
            rc_ptrs, rb_ptrs, nvl_peer_ptrs, csym_peer_ptrs = [], [], [], []

        # varlen metadata: one device buffer, so a layer's descriptors arrive in one copy;
        # cu_q | cu_k | fa_b | fa_mb | fa_order | actv | task table are views at fixed (capacity)
        # offsets, each 16-byte aligned
        def up4(n):
            return (n + 3) // 4 * 4
        # Slots for parts of row tiles' keys: up to SPLIT_HEADS heads' parts (fp32, 65 KB each),
        # and no more than a row tile can have
        slots = min(SPLIT_HEADS // H_local, MAX_PARTS * max_num_row_tiles)
        slots = slots if key_splits and slots >= 2 else 0
        max_tasks = max_num_row_tiles + slots
        sizes = (max_num_batch + 1, max_num_batch + 1, max_num_row_tiles, max_num_row_tiles,
                 max_num_row_tiles, 8, 4 + _cabi.TASK_WORDS * max_tasks)
        offs = [0]
        for n in sizes:
            offs.append(offs[-1] + up4(n))
        meta_dev = zeros(offs[-1], torch.int32)
        mviews = [meta_dev[offs[i]:offs[i] + sizes[i]] for i in range(7)]
        ws = cls(
            dev=dev, dtype=dtype, meta_dev=meta_dev, _meta_offs=offs, tp_size=tp_size, rank=rank, group_name=group_name,
            H_local=H_local, H_kv=H_kv, D=D, K_local=K_local, hidden=hidden,
            hidden_pad=hidden_pad, N_TILE=N_TILE, super_group_n_tiles=super_group_n_tiles,
            q_per_kv=q_per_kv, num_out=num_out, num_super_groups=nsg,
            max_num_row_tiles=max_num_row_tiles, max_num_batch=max_num_batch,
            max_total_oproj=max_total, tot_cap=tot_cap, max_tot_k=max_tot_k,
            paged=bool(paged), page_size=page_size,
            max_num_pages=max_num_pages, max_num_pages_per_seq=max_num_pages_per_seq,
            ctrl=zeros(NUM_CTRL, torch.uint32), sync_ctrl=zeros(NUM_SYNC, torch.uint32),
            actv=mviews[5][:6], status=zeros(NUM_STATUS, torch.uint32),
            head_ready=zeros(max_num_row_tiles, torch.uint32),
            oproj_queue=zeros(max_total, torch.uint32),
            ar_done_bits=zeros(max_owner_words, torch.int64),
            tasks=mviews[6], max_tasks=max_tasks, split_slots=slots,
            parts=torch.empty(slots * H_local * _cabi.PART_FLOATS, dtype=torch.float32, device=dev),
            part_count=zeros(max(slots, 1) * H_local, torch.int32),
            cu_q=mviews[0], cu_k=mviews[1], fa_b=mviews[2], fa_mb=mviews[3], fa_order=mviews[4],
            Q=zeros((tot_cap, H_local, D), dtype),
            K=(None if paged else zeros((max_tot_k, H_kv, D), dtype)),
            V=(None if paged else zeros((max_tot_k, H_kv, D), dtype)),
            K_cache=(zeros((max_num_pages, 128, H_kv, D), dtype) if paged else None),
            V_cache=(zeros((max_num_pages, 128, H_kv, D), dtype) if paged else None),
            page_table=(zeros((max_num_batch, max_num_pages_per_seq), torch.int32)
                        if paged else None),
            cache_seqlens=(zeros(max_num_batch, torch.int32) if paged else None),
            _host_words=(torch.empty(max_num_batch + 2 * _cabi.STEP_BLOCKS, dtype=torch.int32, pin_memory=True).numpy()
                         if paged else None),
            W_o=zeros((K_local, hidden_pad), dtype),
            Oscr=zeros((max_num_row_tiles, 128, H_local, D), dtype),
            csym=csym, rco=rco, rbits=rbits, nvl=nvl,
            csym_mc_ptr=csym_mc_ptr, nvl_peer_ptrs=nvl_peer_ptrs, csym_peer_ptrs=csym_peer_ptrs,
            rc_ptrs=rc_ptrs, rb_ptrs=rb_ptrs, _handles=handles,
        )
        # The first launch relies on every control word being zero on every rank before
        # any rank issues a remote control write.
        torch.cuda.synchronize(dev)
        if tp_size > 1:
            import torch.distributed as dist
            if dist.is_initialized():
                dist.barrier()
        return ws

    # ------------------------------------------------------------------ compile
    def compile(self, w_fa=4, w_oproj=1, w_ar=1, num_ctas=None, kv_stages=2,
                K_CHUNK=64, oproj_stages=4, softmax_scale=None, wait_limit_ms=0, audit=False):
        """Fix the launch configuration and build the C-ABI plan.

        ``kv_stages``, ``K_CHUNK`` and ``oproj_stages`` are accepted for signature
        compatibility; the staging depths of the sm_100a kernel are fixed.
        ``num_ctas=None`` means one CTA per SM.  ``audit=True`` adds execution counters
        (``self.audit``: one per attention (row tile, head), per O_proj slot, per owned
        AllReduce slot; see ``audit_counts``) for exactly-once checks.
        """
        if self._plan is not None:
            self._lib.ma_plan_destroy(self._plan)
            self._plan = None
        # the execution counters exist in the audit build of the library only
        self._lib = _cabi.audit_lib() if audit else _cabi.lib
        d = _cabi.PlanDesc()
        d.device = self.dev.index if self.dev.index is not None else torch.cuda.current_device()
        d.tp_size, d.rank = self.tp_size, self.rank
        d.H_local, d.H_kv, d.D, d.hidden = self.H_local, self.H_kv, self.D, self.hidden
        d.super_group_n_tiles = self.super_group_n_tiles
        d.max_row_tiles, d.max_batch = self.max_num_row_tiles, self.max_num_batch
        d.max_tot_q = self.tot_cap
        d.max_tot_k = self.max_num_pages * 128 if self.paged else self.max_tot_k
        d.softmax_scale = float(softmax_scale) if softmax_scale is not None else 0.0
        d.wait_limit_ms = int(wait_limit_ms)
        kv = (self.K_cache, self.V_cache) if self.paged else (self.K, self.V)
        if self.paged:
            d.page_table = self.page_table.data_ptr()
            d.cache_seqlens = self.cache_seqlens.data_ptr()
            d.max_pages_per_seq = self.max_num_pages_per_seq
        for name, t in (("Q", self.Q), ("K", kv[0]), ("V", kv[1]), ("W_o", self.W_o),
                        ("o_scratch", self.Oscr), ("csym", self.csym), ("ctrl", self.ctrl),
                        ("sync_ctrl", self.sync_ctrl), ("actv", self.actv),
                        ("head_ready", self.head_ready), ("oproj_queue", self.oproj_queue),
                        ("ready_count", self.rco), ("ready_bits", self.rbits),
                        ("ar_done_bits", self.ar_done_bits), ("nvl_signal", self.nvl),
                        ("cu_q", self.cu_q), ("cu_k", self.cu_k), ("fa_b", self.fa_b),
                        ("fa_mb", self.fa_mb), ("status", self.status),
                        ("fa_order", self.fa_order)):
            setattr(d, name, t.data_ptr())
        self.audit = None
        if audit:
            owner_slots = (self.max_total_oproj + self.tp_size - 1) // self.tp_size
            self.audit = torch.zeros(self.max_num_row_tiles * self.H_local + self.max_total_oproj
                                     + owner_slots, dtype=torch.int32, device=self.dev)
            d.audit = self.audit.data_ptr()
        d.csym_multicast = self.csym_mc_ptr
        for r in range(self.tp_size if self.tp_size > 1 else 0):
            d.peer_ready_count[r] = self.rc_ptrs[r]
            d.peer_ready_bits[r] = self.rb_ptrs[r]
            d.peer_nvl_signal[r] = self.nvl_peer_ptrs[r]
            d.peer_csym[r] = self.csym_peer_ptrs[r]
        plan = C.c_void_p()
        _cabi.check(self._lib.ma_plan_create(C.byref(d), C.byref(plan)), "ma_plan_create")
        self._plan = plan
        _cabi.check(self._lib.ma_plan_set_tasks(plan, self.tasks.data_ptr()), "ma_plan_set_tasks")
        if self.split_slots:
            _cabi.check(self._lib.ma_plan_set_split(plan, self.parts.data_ptr(), self.part_count.data_ptr()),
                        "ma_plan_set_split")
        self._split_ctas = int(num_ctas) if num_ctas else torch.cuda.get_device_properties(
            self.dev).multi_processor_count
        self._args = _cabi.LaunchArgs(int(w_fa), int(w_oproj), int(w_ar),
                                      int(num_ctas) if num_ctas else 0, 0)
        self._ts = torch.cuda.current_stream(self.dev)
        self._step_args = None
        return self

    # ------------------------------------------------------------------ per layer
    def set_layer(self, meta, Q, K, V, W_o, page_table=None, cache_seqlens=None):
        """Copy one layer's inputs and varlen metadata into the active prefixes.

        ``Q [tot_q,H_local,D]``, ``K/V [tot_k,H_kv,D]``, ``W_o [K_local,hidden]``; host
        (pinned) or device tensors.  With ``paged=True`` K/V are the caches
        ``[num_pages,128,H_kv,D]`` and ``page_table [B,pps]`` / ``cache_seqlens [B]`` (int32)
        are required.  Raises ``AssertionError`` on any capacity violation before touching
        the workspace.
        """
        R, nb = meta.num_row_tiles, meta.num_batch
        tq = Q.shape[0]
        assert R <= self.max_num_row_tiles and nb <= self.max_num_batch
        assert tq <= self.tot_cap
        assert tuple(Q.shape[1:]) == (self.H_local, self.D)
        assert tuple(W_o.shape) == (self.K_local, self.hidden)
        assert int(meta.cu_seqlens_q[-1]) == tq
        if self.paged:
            # K, V are caches [num_pages, 128, H_kv, D] (workspace.py:213-222 of the reference)
            assert page_table is not None and cache_seqlens is not None
            page_table = torch.as_tensor(page_table, dtype=torch.int32)
            cache_seqlens = torch.as_tensor(cache_seqlens, dtype=torch.int32)
            npg, pps = K.shape[0], page_table.shape[1]
            assert npg <= self.max_num_pages and pps <= self.max_num_pages_per_seq, (
                npg, self.max_num_pages, pps, self.max_num_pages_per_seq)
            assert tuple(K.shape[1:]) == (128, self.H_kv, self.D) == tuple(V.shape[1:])
            assert V.shape[0] == npg and page_table.shape[0] == nb == cache_seqlens.shape[0]
            lens_k = cache_seqlens.cpu().numpy().astype(np.int64)
            lens_q = np.diff(np.asarray(meta.cu_seqlens_q, dtype=np.int64))
            assert bool((lens_k >= lens_q).all()), "q_len > k_len is not supported"
            assert bool((-(-lens_k // 128) <= pps).all())
            assert int(page_table.max()) < npg and int(page_table.min()) >= 0
        else:
            assert page_table is None and cache_seqlens is None
            tk = K.shape[0]
            assert tk <= self.max_tot_k and V.shape[0] == tk
            assert tuple(K.shape[1:]) == (self.H_kv, self.D) == tuple(V.shape[1:])
            assert int(meta.cu_seqlens_k[-1]) == tk
        self._unbind()
        with torch.cuda.stream(self._stream()):
            self.Q[:tq].copy_(Q, non_blocking=True)
            self.W_o[:, :self.hidden].copy_(W_o, non_blocking=True)
            if self.paged:
                self.K_cache[:npg].copy_(K, non_blocking=True)
                self.V_cache[:npg].copy_(V, non_blocking=True)
                self.page_table[:nb, :pps].copy_(page_table.to(self.dev))
                self.cache_seqlens[:nb].copy_(cache_seqlens.to(self.dev))
            else:
                self.K[:tk].copy_(K, non_blocking=True)
                self.V[:tk].copy_(V, non_blocking=True)
            self._set_meta(meta)

    def bind_inputs(self, meta, Q, K, V, W_o, page_table=None, cache_seqlens=None, *,
                    page_table_host=None):
        """Zero-copy alternative to ``set_layer``: the kernel reads the caller's device
        tensors in place (only the varlen metadata is uploaded).  ``W_o`` may be the plain
        ``[K_local, hidden]`` weight when ``hidden % 64 == 0``, else a zero-padded
        ``[K_local, hidden_pad]`` one.  The tensors must stay alive and unchanged until the
        launch has finished; a later ``set_layer`` goes back to the workspace's own buffers.
        """
        R, nb = meta.num_row_tiles, meta.num_batch
        assert R <= self.max_num_row_tiles
        self._check_inputs(nb, int(meta.cu_seqlens_q[-1]), Q, K, V, W_o)
        if self.paged:
            assert page_table is not None and cache_seqlens is not None
            tot_k = K.shape[0] * 128
            page_table = torch.as_tensor(page_table, dtype=torch.int32)
            cache_seqlens = torch.as_tensor(cache_seqlens, dtype=torch.int32)
            assert page_table.shape[1] <= self.max_num_pages_per_seq
            # (the caller may have the page table's values on the host already: one copy of
            # theirs instead of two reductions and two waits for the GPU here)
            pages = page_table if page_table_host is None else page_table_host
            assert int(pages.max()) < K.shape[0] and int(pages.min()) >= 0
        else:
            tot_k = K.shape[0]
            assert int(meta.cu_seqlens_k[-1]) == tot_k
        _cabi.check(self._lib.ma_plan_set_inputs(
            self._plan, Q.data_ptr(), K.data_ptr(), V.data_ptr(), W_o.data_ptr(),
            int(Q.shape[0]), int(tot_k), int(W_o.shape[1])), "ma_plan_set_inputs")
        self._bound = (Q, K, V, W_o)          # keep them alive
        with self._on_stream():
            if self.paged:
                self.page_table[:nb, :page_table.shape[1]].copy_(page_table.to(self.dev))
                self.cache_seqlens[:nb].copy_(cache_seqlens.to(self.dev))
            self._set_meta(meta)

    def _check_inputs(self, nb, tot_q, Q, K, V, W_o):
        """What the kernel can read in place (bind_inputs, step)."""
        for t in (Q, K, V, W_o):
            assert t.is_cuda and t.device == self.dev and t.dtype == self.dtype
            assert t.is_contiguous() and t.data_ptr() % 16 == 0
        assert nb <= self.max_num_batch
        assert Q.shape[1:] == (self.H_local, self.D) and Q.shape[0] <= self.tot_cap
        assert tot_q == Q.shape[0]
        assert W_o.shape[0] == self.K_local and W_o.shape[1] >= self.hidden and W_o.shape[1] % 64 == 0
        want = (128, self.H_kv, self.D) if self.paged else (self.H_kv, self.D)
        assert K.shape[1:] == want == V.shape[1:]
        assert V.shape[0] >= K.shape[0], "V has fewer rows (pages) than K"    # read by K's count

    def can_step(self, *tables):
        """Whether ``step`` takes a call made here and now: one rank, on the stream and device that
        compile() was called on, ``tables`` on that device with columns next to each other."""
        return (self.tp_size == 1 and self._plan is not None
                and torch._C._cuda_getDevice() == self.dev.index == self._ts.device_index
                and torch._C._cuda_getCurrentRawStream(self.dev.index) == self._ts.cuda_stream
                and all(t.device == self.dev and t.stride(-1) == 1 and t.numel() for t in tables))

    def step(self, Q, K, V, W_o, cu_q, cu_k=None, page_table=None, cache_seqlens=None, flags=None):
        """``bind_inputs`` and ``launch`` in one native call (ma_step), for callers whose lengths are
        host arrays (int64 ``cu_q``, ``cu_k``) or, paged, int32 device tensors.  Same refusals.
        Returns the batch's schedule.  Only where ``can_step`` says so."""
        nb = cu_q.size - 1
        self._check_inputs(nb, int(cu_q[-1]), Q, K, V, W_o)
        a = self._step_args
        if a is None:
            a = self._step_args = self._new_step_args()
        if self.paged:
            width = page_table.shape[1]
            assert width <= self.max_num_pages_per_seq
            a.page_table, a.cache_seqlens = page_table.data_ptr(), cache_seqlens.data_ptr()
            a.table_pitch, a.table_width = page_table.stride(0), width
            a.tot_k = K.shape[0] * 128
        else:
            assert cu_k.size == nb + 1 and int(cu_k[-1]) == K.shape[0]
            a.cu_k = cu_k.ctypes.data
            a.tot_k = K.shape[0]
        a.cu_q, a.num_batch = cu_q.ctypes.data, nb
        a.Q, a.K, a.V, a.W_o = Q.data_ptr(), K.data_ptr(), V.data_ptr(), W_o.data_ptr()
        a.tot_q, a.w_width = Q.shape[0], W_o.shape[1]
        prime = self.fa_prime_tiles
        a.stage.meta.auto_prime = int(prime is None)
        a.stage.meta.prime = 0 if prime is None else max(-1, min(int(prime), self.max_num_row_tiles))
        if flags is None:
            flags = self.default_flags or 0      # (launch_flags_b200 is 0 on one rank)
        a.launch.flags = int(flags)
        rc = self._lib.ma_step(self._plan, self._step_at, self._ts.cuda_stream)
        if rc < 0:
            assert rc not in _cabi.STEP_REFUSED, _cabi.STEP_REFUSED[rc]
            _cabi.check(rc, "ma_step")
        self._bound = (Q, K, V, W_o, page_table)      # keep them alive
        self._auto_flags = 0
        self._meta = StepMeta(cu_q, self._host_words[:nb] if self.paged else None, cu_k, rc)
        return self._meta

    def _new_step_args(self):
        """The part of ma_step's arguments that is the workspace's."""
        if getattr(self, "_meta_host", None) is None:
            self._meta_host = np.zeros(self._meta_offs[-1], dtype=np.int32)
            self._meta_at = self._meta_host.ctypes.data
        o = self._meta_offs
        a = _cabi.StepArgs()
        a.stage = _cabi.StageTasksArgs(_cabi.StageMetaArgs(
            None, None, None, None, self._meta_at, 0, 0, self.hidden, self.H_local, self.num_super_groups,
            self.tp_size, self.rank, 1, 0, o[0], o[1], o[2], o[3], o[4], o[5], 0), o[6], self.max_tasks,
            self.split_slots, self._split_ctas)
        a.meta_dev, a.max_row_tiles, a.launch = self.meta_dev.data_ptr(), self.max_num_row_tiles, self._args
        if self.paged:
            a.page_table_out, a.cache_seqlens_out = self.page_table.data_ptr(), self.cache_seqlens.data_ptr()
            a.table_pitch_out, a.host_words = self.max_num_pages_per_seq, self._host_words.ctypes.data
        self._step_at = C.addressof(a)
        return a

    def _unbind(self):
        if getattr(self, "_bound", None) is not None:
            kv = (self.K_cache, self.V_cache) if self.paged else (self.K, self.V)
            tot_k = self.max_num_pages * 128 if self.paged else self.max_tot_k
            _cabi.check(self._lib.ma_plan_set_inputs(
                self._plan, self.Q.data_ptr(), kv[0].data_ptr(), kv[1].data_ptr(),
                self.W_o.data_ptr(), self.tot_cap, tot_k, self.hidden_pad), "ma_plan_set_inputs")
            self._bound = None

    def set_meta(self, meta):
        """Metadata only (inputs already resident in ``self.Q/K/V/W_o``)."""
        assert meta.num_row_tiles <= self.max_num_row_tiles
        assert meta.num_batch <= self.max_num_batch
        assert int(meta.cu_seqlens_q[-1]) <= self.tot_cap
        assert self.paged or int(meta.cu_seqlens_k[-1]) <= self.max_tot_k
        with torch.cuda.stream(self._stream()):
            self._set_meta(meta)

    def _set_meta(self, meta):
        R = meta.num_row_tiles
        # (the words travel in a kernel's parameters, so the staging copy is free again on return)
        if getattr(self, "_meta_host", None) is None:
            self._meta_host = np.zeros(self._meta_offs[-1], dtype=np.int32)
            self._meta_at = self._meta_host.ctypes.data
        o = self._meta_offs
        self._auto_flags = launch_flags_b200(meta, self.hidden, self.tp_size, self.H_local)
        cu_q, cu_k, b_idx, m_blk = (np.ascontiguousarray(x, dtype=np.int32) for x in (
            meta.cu_seqlens_q, meta.cu_seqlens_k, meta.batch_idx, meta.m_block))
        assert b_idx.size == m_blk.size == R and cu_q.size == cu_k.size == meta.num_batch + 1
        prime = self.fa_prime_tiles
        args = _cabi.StageTasksArgs(_cabi.StageMetaArgs(
            cu_q.ctypes.data, cu_k.ctypes.data, b_idx.ctypes.data, m_blk.ctypes.data,
            self._meta_at, cu_q.size - 1, R, self.hidden, self.H_local, self.num_super_groups,
            self.tp_size, self.rank, int(prime is None),
            0 if prime is None else max(-1, min(int(prime), R)),
            o[0], o[1], o[2], o[3], o[4], o[5], 0), o[6], self.max_tasks, self.split_slots,
            self._split_ctas)
        rc = _cabi.lib.ma_upload_meta(C.byref(args), self.meta_dev.data_ptr(),
                                      torch.cuda.current_stream(self.dev).cuda_stream)
        _cabi.check(min(rc, 0), "ma_upload_meta")
        self._meta = meta

    def _on_stream(self):
        """``torch.cuda.stream(self._stream())``, or nothing to do if that is current (device
        included): the usual case, and a fifth of a small step's host time."""
        st = self._stream()
        if torch.cuda.current_stream() == st:
            return contextlib.nullcontext()
        return torch.cuda.stream(st)

    def _stream(self):
        return getattr(self, "_ts", None) or torch.cuda.current_stream(self.dev)

    def launch(self, flags=None):
        assert self._plan is not None, "call compile() first"
        if flags is None:
            flags = self._auto_flags if self.default_flags is None else self.default_flags
        if self.tp_size == 2 and self.ar_p2p:
            # two GPUs: reduce with peer loads/stores, not multimem (see MA_FLAG_AR_P2P)
            flags |= _cabi.MA_FLAG_AR_P2P
        args = _cabi.LaunchArgs(self._args.w_fa, self._args.w_oproj, self._args.w_ar,
                                self._args.num_ctas, int(flags))
        _cabi.check(self._lib.ma_launch(self._plan, C.byref(args),
                                        C.c_void_p(self._ts.cuda_stream)), "ma_launch")

    def launch_fa_only(self):
        """Attention stage alone (fills ``Oscr``); used by the unfused baseline."""
        self.launch(flags=_cabi.MA_FLAG_FA_ONLY)

    def launch_oproj_only(self):
        """O_proj stage alone (single rank): ``Oscr`` must hold a finished attention output."""
        assert self.tp_size == 1
        self.launch(flags=_cabi.MA_FLAG_OPROJ_ONLY)

    def launch_ar_only(self, extra_flags=0):
        """AllReduce stage alone over every slot of ``csym`` (tp > 1).  Every rank's partial
        must be complete before any rank launches (e.g. after a host barrier)."""
        assert self.tp_size > 1, "the AllReduce stage needs tp_size > 1"
        self.launch(flags=_cabi.MA_FLAG_AR_ONLY | extra_flags)

    def audit_counts(self, meta=None):
        """``(attention [R, H_local], o_proj [R * nsg], allreduce [owned])`` execution
        counts since the last ``audit.zero_()`` (``compile(audit=True)``)."""
        meta = meta or self._meta
        R = meta.num_row_tiles
        a = self.audit.cpu()
        n_fa, n_op = self.max_num_row_tiles * self.H_local, self.max_total_oproj
        total = R * self.num_super_groups
        owned = max(total - self.rank, 0)
        owned = (owned + self.tp_size - 1) // self.tp_size
        return (a[:R * self.H_local].view(R, self.H_local), a[n_fa:n_fa + total],
                a[n_fa + n_op:n_fa + n_op + owned])

    def check_status(self):
        """Synchronise the launch stream and raise if a device-side wait gave up."""
        st = _cabi.Status()
        rc = self._lib.ma_read_status(self._plan, C.c_void_p(self._ts.cuda_stream), C.byref(st))
        if rc != _cabi.MA_OK:
            raise RuntimeError(
                f"fused prefill kernel: {_cabi.strerror(rc)} "
                f"(code={st.code} site=0x{st.site:x} cta={st.cta} aux={st.aux}); "
                "the workspace control state is undefined — call debug_zero_all()")

    def output(self, meta=None):
        """De-tiled ``[tot_q, hidden]`` copy of the valid region of ``csym``, queued on the
        current stream."""
        meta = meta or self._meta
        cu_q = np.ascontiguousarray(meta.cu_seqlens_q, dtype=np.int32)
        assert meta.num_row_tiles <= self.max_num_row_tiles
        out = torch.empty(int(cu_q[-1]), self.hidden, dtype=self.dtype, device=self.dev)
        args = _cabi.DetileArgs(self.csym.data_ptr(), out.data_ptr(), cu_q.ctypes.data,
                                cu_q.size - 1, self.hidden, self.hidden_pad, 0)
        with torch.cuda.device(self.dev):
            _cabi.check(self._lib.ma_detile(
                C.byref(args), C.c_void_p(torch.cuda.current_stream(self.dev).cuda_stream)),
                "ma_detile")
        return out

    # ------------------------------------------------------------------ debug
    def debug_zero_all(self):
        """Fault localisation only; never on the production / bench / test default path.
        With tp > 1 every rank must call it, followed by a host barrier."""
        for t in (self.ctrl, self.sync_ctrl, self.actv, self.head_ready, self.oproj_queue,
                  self.fa_order, self.tasks, self.part_count, self.rco, self.rbits, self.ar_done_bits, self.nvl, self.csym, self.Oscr,
                  self.status):
            t.zero_()

    def __del__(self):
        try:
            if self._plan is not None:
                self._lib.ma_plan_destroy(self._plan)
                self._plan = None
        except Exception:
            pass
