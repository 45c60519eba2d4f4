"""Per-rank device state and thin launch wrappers around the native kernels.

Every wrapper takes LISTS (one entry per rank hosted by this process): a normal
``Buffer`` passes lists of length one; the single-GPU ``LocalCluster`` passes all R ranks
so that one cooperative launch runs every rank's CTAs side by side (blockIdx.y = rank)
and the cross-rank barriers work on one device.
"""

from __future__ import annotations

import ctypes as C
import os
from dataclasses import dataclass, field

import torch

from . import _native
from ._native import (MepRankCtx, PlanArgs, DispatchArgs, DupFinalizeArgs, DupArgs, CombineArgs, PushReduceArgs,
                      PrefetchArgs, GradReduceArgs, SendOrderArgs, ptr)
from .geometry import Geometry
from .plan import MoonEPCommPlan

ERROR_NAMES = {1: "grid barrier timed out (a CTA never arrived)",
               2: "cross-rank barrier timed out (a peer never arrived)",
               3: "index out of range",
               4: "ready flag never reached its expected value",
               5: "mbarrier phase never completed"}
KERNEL_NAMES = {1: "rank_sync", 2: "planning", 3: "dispatch", 4: "dup_expand", 5: "dup_reduce", 6: "combine",
                7: "prefetch", 8: "grad_reduce", 9: "grouped_gemm", 10: "wait_probe"}


LOCAL_MAX_E = 2048


class MoonEPTimeout(RuntimeError):
    """A bounded device-side wait expired (or a checked index was out of range)."""

    def __init__(self, status: dict):
        self.status = status
        super().__init__(
            f"rank {status['rank']}: {KERNEL_NAMES.get(status['kernel'], status['kernel'])} kernel, site "
            f"{status['site']}: {ERROR_NAMES.get(status['code'], status['code'])} "
            f"(peer/cta {status['peer']}, observed {status['observed']}, expected {status['expected']})")


def wait_budget_ns() -> int:
    ms = float(os.environ.get("MOONEP_WAIT_BUDGET_MS", "2000"))
    return max(1, int(ms * 1e6))


@dataclass
class RankState:
    geo: Geometry
    rank: int
    heap: object
    device: torch.device
    ctx_host: MepRankCtx = None
    ctx_dev: torch.Tensor = None
    scratch: dict = field(default_factory=dict)
    hidden_local: torch.Tensor = None     # [NvS, H] bf16 view of this rank's shard
    weights_local: torch.Tensor = None    # [NvS] fp32 view
    srcinfo_local: torch.Tensor = None    # [NvS] int32 provenance table (push-combine Buffers only)
    status: torch.Tensor = None           # int32[8] device
    status_host: torch.Tensor = None      # int32[1] pinned host memory the kernels mirror status[0] into
    plan_fast: bool = False
    local: bool = False                   # single rank: dispatch / combine are one local kernel each
    local_blocks: int = 0                 # CTAs the local dispatch has scratch for

    @property
    def ctx_ptr(self) -> int:
        return self.ctx_dev.data_ptr()


def make_rank_state(geo: Geometry, rank: int, heap, device, budget_ns: int | None = None) -> RankState:
    dev = torch.device(device)
    st = RankState(geo, rank, heap, dev)
    i32 = dict(dtype=torch.int32, device=dev)
    R, E, epn = geo.R, geo.E, geo.epn
    s = st.scratch
    s["grid_bar"] = torch.zeros(4, **i32)
    s["epoch"] = torch.zeros(_native.BAR_ROWS, **i32)
    s["hist"] = torch.zeros(geo.num_vblocks * E, **i32)
    s["vb_flags"] = torch.zeros(geo.num_vblocks + 2, **i32)      # + the fast planner's epoch word and exit counter
    s["count"] = torch.zeros(E, **i32)
    s["tpe_prefix"] = torch.zeros(E, **i32)
    s["remaining"] = torch.zeros(E, **i32)
    s["alloc"] = torch.zeros(E * R, **i32)
    s["alloc_cumsum"] = torch.zeros(E * R, **i32)
    s["expert_off"] = torch.zeros(R * E, **i32)
    s["etc_all"] = torch.zeros(R * epn, **i32)
    s["stats_all"] = torch.zeros(R * 2, **i32)
    s["send_cnt"] = torch.zeros(2 * R, dtype=torch.int64, device=dev)     # two halves, see planning_fast_kernel
    s["tile_done"] = torch.zeros(geo.ntiles, **i32)           # ready flags: epoch at which a tile became complete
    s["flag_epoch"] = torch.zeros(4, **i32)                   # [0] flagged dispatches issued, [1] expander ticket
    s["slot_done"] = torch.zeros(R * epn, **i32)              # prefetch: chunks finished per (rank, slot), self-resetting
    s["pf_epoch"] = torch.zeros(2, **i32)                     # prefetch launches issued
    if os.environ.get("MOONEP_COUNTERS", "1") != "0":
        s["counters"] = torch.zeros(_native.COUNTER_SLOTS, dtype=torch.int64, device=dev)
    checked = os.environ.get("MOONEP_CHECKED") == "1"
    # a group of one rank exchanges rows with nobody: see csrc/device/local_exchange.cu. The checked mode keeps the
    # general kernels (its table checks sit between them); E is what the kernel's tables in shared memory hold.
    st.local = R == 1 and E <= LOCAL_MAX_E and not checked
    if st.local:
        st.local_blocks = torch.cuda.get_device_properties(dev).multi_processor_count
        s["loc_sync"] = torch.zeros(16 + st.local_blocks, **i32)
        s["loc_hist"] = torch.empty(st.local_blocks * E, **i32)
    st.status = torch.zeros(8, **i32)
    # first failure code, mirrored by the kernels into host memory the device can write: the host
    # tests it without synchronising (see Buffer._st)
    st.status_host = torch.zeros(1, dtype=torch.int32).pin_memory()

    c = MepRankCtx()
    c.rank, c.R, c.S, c.H, c.K, c.E, c.epn, c.N, c.NvS = rank, R, geo.S, geo.H, geo.K, E, epn, geo.N, geo.NvS
    c.token_padding, c.vblock_entries, c.num_vblocks = geo.token_padding, geo.vblock_entries, geo.num_vblocks
    c.num_sms = geo.num_sms
    c.checked = 1 if checked else 0
    c.heap_base, c.chunk_stride = heap.base, heap.chunk_bytes
    for name in ("off_hidden", "off_weights", "off_tpe", "off_bar", "off_dupcnt", "off_dupgroups",
                 "off_duploffs", "off_ready", "off_rowsrc", "off_slotflag"):
        setattr(c, name, getattr(geo, name))
    c.dup_group_cap, c.dup_loff_cap = geo.dup_group_cap, geo.dup_loff_cap
    for name in ("grid_bar", "epoch", "hist", "count", "tpe_prefix", "remaining", "alloc", "alloc_cumsum",
                 "expert_off", "etc_all", "stats_all", "send_cnt", "vb_flags", "tile_done", "flag_epoch", "slot_done",
                 "pf_epoch"):
        setattr(c, name, s[name].data_ptr())
    c.ntiles = geo.ntiles
    c.counters = s["counters"].data_ptr() if "counters" in s else None
    c.status = st.status.data_ptr()
    c.status_host = st.status_host.data_ptr()
    c.wait_budget_ns = wait_budget_ns() if budget_ns is None else budget_ns
    c.mc_base = getattr(heap, "mc_base", 0) or None
    if os.environ.get("MOONEP_TRACE") == "1":
        cap = int(os.environ.get("MOONEP_TRACE_RECORDS", "65536"))
        s["trace"] = torch.zeros(1 + 2 * cap, dtype=torch.int64, device=dev)
        c.trace, c.trace_cap = s["trace"].data_ptr(), cap
    st.ctx_host = c
    st._failed_word = C.c_int32.from_address(st.status_host.data_ptr())
    raw = bytes(c)
    st.ctx_dev = torch.frombuffer(bytearray(raw), dtype=torch.uint8).to(dev)
    st.plan_fast = bool(_native.load().mep_planning_is_fast(E, R))
    st.hidden_local = heap.view(rank, geo.off_hidden, (geo.NvS, geo.H), torch.bfloat16)
    st.weights_local = heap.view(rank, geo.off_weights, (geo.NvS,), torch.float32)
    st.srcinfo_local = heap.view(rank, geo.off_srcinfo, (geo.NvS,), torch.int32) if geo.off_srcinfo else None
    return st


def failed(st: RankState) -> bool:
    """True once any kernel of this rank has recorded a failure. A plain read of host memory: no
    synchronisation, usable between launches and during CUDA-graph replays."""
    return st._failed_word.value != 0


def read_counters(st: RankState, reset: bool = False) -> dict:
    """Per-op device counters accumulated since the Buffer was created or last reset (synchronises)."""
    t = st.scratch.get("counters")
    if t is None:
        return {}
    v = t.cpu().tolist()
    out = {name: int(v[i]) for i, name in _native.COUNTER_NAMES.items()}
    out["rows_sent_to"] = [int(x) for x in v[_native.COUNTER_PEER_BASE:_native.COUNTER_PEER_BASE + min(st.geo.R, 48)]]
    if reset:
        t.zero_()
    return out


def read_status(st: RankState) -> dict | None:
    v = st.status.cpu().tolist()
    if v[0] == 0:
        return None
    return dict(code=v[0], kernel=v[1], site=v[2], rank=v[3], peer=v[4],
                observed=v[5] & 0xFFFFFFFF, expected=v[6] & 0xFFFFFFFF)


def read_trace(st: RankState, reset: bool = True):
    """Device timestamps recorded since the last reset: list of ``(ns, kernel, site, cta, warp)``
    sorted by time (needs ``MOONEP_TRACE=1`` when the Buffer was created). Synchronises."""
    t = st.scratch.get("trace")
    if t is None:
        return []
    v = t.cpu()
    n = min(int(v[0]), (v.numel() - 1) // 2)
    out = []
    for i in range(n):
        ns, tag = int(v[1 + 2 * i]), int(v[2 + 2 * i])
        out.append((ns, (tag >> 48) & 0xFFFF, (tag >> 32) & 0xFFFF, (tag >> 8) & 0xFFFFFF, tag & 0xFF))
    if reset:
        t[0] = 0
    return sorted(out)


def _pack(states):
    return _native.ctx_array([s.ctx_ptr for s in states])


def allocate_plan(st: RankState, with_send_list: bool = False):
    """Plan-owned tensors plus cu_seqlens for one rank (reference: planning.py:1168-1215).  They are views of ONE
    allocation, each starting on a 16-byte boundary: a plan costs one allocator call instead of eight, which is
    what a small dispatch would otherwise wait for."""
    sizes, total, _ = _plan_layout(st, with_send_list)
    parts = torch.empty(total, dtype=torch.int32, device=st.device).split(sizes)[::2]
    if not st.local:
        parts[6].zero_()
    if with_send_list:
        parts[9].zero_()
    return _plan_of_parts(st.geo, parts, with_send_list)


def _plan_layout(st: RankState, with_send_list: bool = False):
    """``(sizes and gaps, total, first element of every field)`` of a plan's allocation."""
    key = "plan_layout_send" if with_send_list else "plan_layout"
    lay = st.scratch.get(key)
    if lay is None:
        g = st.geo
        sizes = [g.N, g.R * g.epn, 4 * g.epn, 2, 3 * g.NvS, g.NvS, 2, 2 * g.epn] + ([g.N, 4] if with_send_list else [])
        both, first, off = [], [], 0
        for n in sizes:
            first.append(off)
            both += [n, -n % 4]
            off += n + -n % 4
        lay = st.scratch[key] = (both, off, first)
    return lay


def _plan_of_parts(g: Geometry, parts, with_send_list: bool = False):
    extra = dict(send_list=parts[8], send_meta=parts[9]) if with_send_list else {}
    plan = MoonEPCommPlan.of_parts(
        dst=parts[0], experts_to_copy=parts[1].view(g.R, g.epn), zero_fill_ranges=parts[2].view(2 * g.epn, 2),
        remote_stats=parts[3], N=g.N, R=g.R, E=g.E, NvS=g.NvS, K=g.K,
        dup_groups=parts[4].view(g.NvS, 3), dup_loffs=parts[5], dup_counts=parts[6], **extra)
    return plan, parts[7]


class LocalExchange:
    """Single-rank dispatch and combine, one native call each (csrc/host/moe_local.cc)."""

    def __init__(self, st: RankState, blocks: int):
        g, a = st.geo, _native.MoeLocal()
        a.ctx = st.ctx_ptr
        a.S, a.H, a.K, a.E, a.NvS, a.token_padding = g.S, g.H, g.K, g.E, g.NvS, g.token_padding
        a.blocks, a.combine_blocks, a.sms = min(blocks, st.local_blocks), blocks, st.local_blocks
        _, self._total, first = _plan_layout(st)
        a.plan_off = (C.c_int64 * 8)(*first)
        self._cu_first, self._cu_shape = first[7], (2 * g.epn,)
        a.shard, a.shard_w, a.srcinfo = st.hidden_local.data_ptr(), st.weights_local.data_ptr(), ptr(st.srcinfo_local)
        a.sync, a.hist = st.scratch["loc_sync"].data_ptr(), st.scratch["loc_hist"].data_ptr()
        self._args, self._ref, self._dev = a, C.addressof(a), st.device
        # the block of a combine whose rows a saved plan has brought (an argument for it and
        # its lookup cost a decode batch of 64 0.4 us of 23.4)
        self._args_in_order = _native.MoeLocal.from_buffer_copy(a)
        self._args_in_order.in_order = 1
        self._ref_in_order = C.addressof(self._args_in_order)
        self.pdl = False                    # see set_pdl
        self._ints = dict(N=g.N, R=g.R, E=g.E, NvS=g.NvS, K=g.K)
        # shape, strides and first element of each part: one as_strided call costs a third of narrow and view
        self._fields = dict(dst=((g.N,), (1,), first[0]), experts_to_copy=((1, g.epn), (g.epn, 1), first[1]),
                            zero_fill_ranges=((2 * g.epn, 2), (2, 1), first[2]), remote_stats=((2,), (1,), first[3]),
                            dup_groups=((g.NvS, 3), (3, 1), first[4]), dup_loffs=((g.NvS,), (1,), first[5]), dup_counts=((2,), (1,), first[6]))
        # what results are made like: half the cost of a size, a type and a device
        self._rows_like = st.hidden_local.narrow(0, 0, g.S)
        self._weights_like = st.weights_local.as_strided((g.S, g.K), (g.K, 1))
        self._lib = _native.load()

    def set_pdl(self, pdl: bool):
        """Whether a call's kernel may set itself up while the kernel before it in the stream still runs."""
        self.pdl = self._args.pdl = self._args_in_order.pdl = bool(pdl)

    def _name_part(self, slab, name):
        f = self._fields.get(name)
        if f is None:
            return None
        return slab.as_strided(*f)

    def plan_of(self, slab):
        """``(plan, cu_seqlens)`` of an allocation that a native call has planned into."""
        return MoonEPCommPlan.of_slab(slab, self._name_part, self._ints), slab.as_strided(self._cu_shape, (1,), self._cu_first)

    def dispatch(self, hidden, route_w, topk, tpe, out_hidden, out_w):
        """A fresh plan (in one allocation: what a small dispatch would otherwise wait for) and the K rows of every
        token; returns ``(plan, cu_seqlens)``.  ``out_hidden`` / ``out_w``: any tensors of the shard's shape."""
        slab = torch.empty(self._total, dtype=torch.int32, device=self._dev)
        rc = self._lib.mep_local_dispatch_call(self._ref, hidden.data_ptr(), None if route_w is None else route_w.data_ptr(),
                                               topk.data_ptr(), tpe.data_ptr(), slab.data_ptr(), None, None, out_hidden.data_ptr(),
                                               None if out_w is None else out_w.data_ptr(), _native.raw_stream())
        if rc:
            _native.check(rc, "dispatch")
        return self.plan_of(slab)

    def dispatch_again(self, hidden, route_w, plan, out_hidden, out_w):
        """The rows of a saved plan."""
        plan.__dict__["_in_order"] = True   # a hint for the combine of these rows; either order gives the same sums
        rc = self._lib.mep_local_dispatch_call(self._ref, hidden.data_ptr(), None if route_w is None else route_w.data_ptr(), None, None,
                                               None, self._dst(plan), plan.zero_fill_ranges.data_ptr(), out_hidden.data_ptr(),
                                               None if out_w is None else out_w.data_ptr(), _native.raw_stream())
        if rc:
            _native.check(rc, "dispatch")

    @staticmethod
    def _dst(plan) -> int:      # the first field of a plan's allocation
        slab = plan.__dict__.get("_slab")
        return plan.dst.data_ptr() if slab is None else slab.data_ptr()

    def combine(self, plan, rows, row_w):
        """``(out, out_w)``: ``out[s]`` = sum of the K rows of token ``s``; ``rows`` / ``row_w`` are any tensors of the shard's shape and only
        read."""
        out = torch.empty_like(self._rows_like)
        out_w = None if row_w is None else torch.empty_like(self._weights_like)
        d = plan.__dict__
        slab = d.get("_slab")
        rc = self._lib.mep_local_combine_call(self._ref_in_order if "_in_order" in d else self._ref,
                                              plan.dst.data_ptr() if slab is None else slab.data_ptr(), rows.data_ptr(), None if row_w is None else row_w.data_ptr(),
                                              out.data_ptr(), None if out_w is None else out_w.data_ptr(), _native.raw_stream())
        if rc:
            _native.check(rc, "combine")
        return out, out_w


class LocalLayer(LocalExchange):
    """A single-rank MoE layer's forward and backward pass as one native call each (csrc/host/moe_local.cc).  ``work``:
    the layer's own buffers.  The addresses of weights and gradients (gate, up, down) come with every call."""

    def __init__(self, st: RankState, Hp: int, work: dict, blocks: int, num_ctas: int, status, status_host, budget_ns: int):
        super().__init__(st, blocks)
        self.state = st
        self._weights, self._grads, self._pdl = (None,) * 3, (None,) * 3, None      # what the argument block holds
        a = self._args
        a.Hp, a.num_ctas = Hp, num_ctas
        for name, t in work.items():
            setattr(a, name, t.data_ptr())
        a.status, a.status_host, a.budget_ns = status.data_ptr(), status_host.data_ptr(), budget_ns

    def _set(self, weights, grads, pdl):
        if weights != self._weights or grads != self._grads or pdl != self._pdl:
            a = self._args
            a.w_gate, a.w_up, a.w_down = self._weights = weights
            a.dw_gate, a.dw_up, a.dw_down = self._grads = grads
            a.pdl = self._pdl = pdl

    def forward(self, hidden, route_w, topk, tpe, keep: bool, weights, pdl: bool):
        """Returns ``(out, plan allocation)``."""
        self._set(weights, self._grads, pdl)
        slab = torch.empty(self._total, dtype=torch.int32, device=self._dev)
        out = torch.empty_like(self._rows_like)
        rc = self._lib.mep_moe_local_forward(self._ref, hidden.data_ptr(), route_w.data_ptr(), topk.data_ptr(), tpe.data_ptr(),
                                             slab.data_ptr(), out.data_ptr(), 1 if keep else 0, _native.raw_stream())
        if rc:
            _native.check(rc, "moe forward")
        return out, slab

    def backward(self, dy, slab, accumulate: bool, lr: float, mask, weights, grads, pdl: bool):
        self._set(weights, grads, pdl)
        dx, dw = torch.empty_like(self._rows_like), torch.empty_like(self._weights_like)
        rc = self._lib.mep_moe_local_backward(self._ref, dy.data_ptr(), slab.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                              1 if accumulate else 0, lr, ptr(mask), _native.raw_stream())
        if rc:
            _native.check(rc, "moe backward")
        return dx, dw


def launch_planning(states, topk_list, tpe_list, plans, cu_list):
    lib = _native.load()
    n = len(states)
    args = (PlanArgs * n)()
    for i in range(n):
        p = plans[i]
        st = states[i]
        args[i] = PlanArgs(ptr(topk_list[i]), ptr(tpe_list[i]), ptr(p.dst), ptr(cu_list[i]),
                           ptr(p.experts_to_copy), ptr(p.zero_fill_ranges), ptr(p.remote_stats),
                           1 if st.plan_fast else 0, 0)
    g = states[0].geo
    _native.check(lib.mep_launch_planning(n, _pack(states), args, g.num_sms, g.E, g.R, _native.cur_stream()), "planning")


def launch_dispatch(states, hidden_list, weights_list, plans, fresh: bool, entry_barrier: bool, flagged: bool = False):
    lib = _native.load()
    n = len(states)
    g0 = states[0].geo
    args = (DispatchArgs * n)()
    for i in range(n):
        w = weights_list[i] if weights_list is not None else None
        fresh_code = 3 if states[i].plan_fast else 1      # which send_cnt half the planner used (3: device epoch)
        args[i] = DispatchArgs(ptr(hidden_list[i]), ptr(w), ptr(plans[i].dst), ptr(plans[i].zero_fill_ranges),
                               fresh_code if fresh else 0, 1 if entry_barrier else 0, g0.off_srcinfo,
                               ptr(plans[i].send_list), ptr(plans[i].send_meta))
    g = states[0].geo
    fn = lib.mep_launch_dispatch_flagged if flagged else lib.mep_launch_dispatch
    _native.check(fn(n, _pack(states), args, g.num_sms, g.H, g.epn, _native.cur_stream()), "dispatch")


def launch_send_order(states, plans, cu_list):
    """Build each plan's send list (``plan.send_list`` / ``plan.send_meta``) from ``plan.dst``."""
    lib = _native.load()
    n = len(states)
    args = (SendOrderArgs * n)()
    g = states[0].geo
    for i in range(n):
        sc = states[i].scratch
        if "send_hist" not in sc:       # bucket histogram and per-entry bucket, sized on first use
            nb = lib.mep_send_order_buckets(g.NvS, g.R, None)
            sc["send_hist"] = torch.zeros(nb, dtype=torch.int32, device=states[i].device)
            sc["send_bucket"] = torch.empty(g.N, dtype=torch.int32, device=states[i].device)
        args[i] = SendOrderArgs(ptr(plans[i].dst), ptr(cu_list[i]), ptr(plans[i].send_list), ptr(plans[i].send_meta),
                                ptr(sc["send_hist"]), ptr(sc["send_bucket"]))
    _native.check(lib.mep_launch_send_order(n, _pack(states), args, g.N, g.NvS, g.R, _native.cur_stream()), "send_order")


def launch_flag_epoch_bump(states):
    """A flagged dispatch is about to be issued: advance the flag epoch on the current stream, ahead
    of the dispatch kernel and of every consumer of its tile flags."""
    lib = _native.load()
    _native.check(lib.mep_launch_flag_epoch_bump(len(states), _pack(states), _native.cur_stream()), "flag_epoch_bump")


def launch_tile_wait_probe(st: RankState, tile: int):
    lib = _native.load()
    _native.check(lib.mep_launch_tile_wait_probe(C.c_void_p(st.ctx_ptr), tile, _native.cur_stream()), "tile_wait_probe")


def launch_dup_finalize(states, plans):
    lib = _native.load()
    n = len(states)
    args = (DupFinalizeArgs * n)()
    for i in range(n):
        args[i] = DupFinalizeArgs(ptr(plans[i].dup_groups), ptr(plans[i].dup_loffs), ptr(plans[i].dup_counts))
    _native.check(lib.mep_launch_dup_finalize(n, _pack(states), args, _native.cur_stream()), "dup_finalize")


def launch_dup_expand_fresh(states, bufs, plans, num_blocks: int, pdl: bool = False):
    """Fresh dispatch: compact the staged duplicate groups into the plan and expand them, one launch.
    ``pdl``: programmatic dependent launch behind the kernel queued just before on this stream."""
    lib = _native.load()
    _native.check(lib.mep_launch_dup_expand_fresh(len(states), _pack(states), _dup_args(states, bufs, plans),
                                                  num_blocks, 1 if pdl else 0, _native.cur_stream()), "dup_expand_fresh")


def _dup_args(states, bufs, plans):
    n = len(states)
    args = (DupArgs * n)()
    for i in range(n):
        args[i] = DupArgs(ptr(bufs[i]), ptr(plans[i].dup_groups), ptr(plans[i].dup_loffs), ptr(plans[i].dup_counts))
    return args


def _dup_check(states, bufs, plans, num_blocks: int, kernel_id: int):
    """MOONEP_CHECKED=1: validate the duplicate tables in a pass of their own before they are used."""
    if states[0].ctx_host.checked:
        lib = _native.load()
        _native.check(lib.mep_launch_dup_check(len(states), _pack(states), _dup_args(states, bufs, plans), num_blocks,
                                               kernel_id, _native.cur_stream()), "dup_check")


def launch_dup_expand(states, bufs, plans, num_blocks: int, pdl: bool = False):
    lib = _native.load()
    _dup_check(states, bufs, plans, num_blocks, 4)
    pdl = pdl and not states[0].ctx_host.checked        # the check sits between dispatch and this kernel
    _native.check(lib.mep_launch_dup_expand(len(states), _pack(states), _dup_args(states, bufs, plans),
                                            num_blocks, 1 if pdl else 0, _native.cur_stream()), "dup_expand")


def launch_dup_reduce(states, bufs, plans, num_blocks: int):
    lib = _native.load()
    _dup_check(states, bufs, plans, num_blocks, 5)
    _native.check(lib.mep_launch_dup_reduce(len(states), _pack(states), _dup_args(states, bufs, plans),
                                            num_blocks, _native.cur_stream()), "dup_reduce")


def launch_combine(states, plans, outs, out_weights, entry_barrier: bool = True, pdl: bool = False):
    lib = _native.load()
    n = len(states)
    args = (CombineArgs * n)()
    for i in range(n):
        ow = out_weights[i] if out_weights is not None else None
        args[i] = CombineArgs(ptr(plans[i].dst), ptr(outs[i]), ptr(ow), 1 if entry_barrier else 0)
    _native.check(lib.mep_launch_combine(n, _pack(states), args, states[0].geo.num_sms, 1 if pdl else 0, _native.cur_stream()), "combine")


def launch_rank_sync(states):
    lib = _native.load()
    _native.check(lib.mep_launch_rank_sync(len(states), _pack(states), _native.cur_stream()), "rank_sync")


def _rank_stride_bytes(pool: torch.Tensor) -> int:
    return int(pool.stride(0)) * pool.element_size()


def launch_pf_epoch_bump(states):
    """A prefetch is about to be issued: advance the prefetch epoch.  Must run in stream order before the
    prefetch kernel AND before any GEMM that waits on its slot flags, i.e. on the stream both are forked from."""
    lib = _native.load()
    _native.check(lib.mep_launch_pf_epoch_bump(len(states), _pack(states), _native.cur_stream()), "pf_epoch_bump")


def launch_prefetch(states, etc_list, tensor_pairs_list, bump_epoch: bool = True):
    """``tensor_pairs_list[i]`` = sequence of up to six ``(local[epn,...], pool[R,epn,...])``.
    ``bump_epoch=False``: the caller has already advanced the prefetch epoch (``launch_pf_epoch_bump``)."""
    lib = _native.load()
    n = len(states)
    args = (PrefetchArgs * n)()
    for i in range(n):
        a = PrefetchArgs()
        a.etc = ptr(etc_list[i])
        pairs = tensor_pairs_list[i]
        a.ntensors = len(pairs)
        for j, (local, pool) in enumerate(pairs):
            a.t[j].local = local.data_ptr()
            a.t[j].pool = pool.data_ptr()
            a.t[j].expert_bytes = local[0].numel() * local.element_size()
            a.t[j].rank_stride = _rank_stride_bytes(pool)
        args[i] = a
    g = states[0].geo
    # new prefetch epoch first (stream order): the kernel stamps completed slots with it and a GEMM that
    # consumes the slots while the prefetch runs compares against it
    if bump_epoch:
        launch_pf_epoch_bump(states)
    _native.check(lib.mep_launch_prefetch(n, _pack(states), args, g.num_sms, g.R, g.epn, _native.cur_stream()), "prefetch")


def launch_grad_reduce(states, etc_list, tensor_pairs_list, entry_barrier: bool = True, clear_slots: bool = True):
    """``entry_barrier``: wait for every rank before the first peer read (the holders' weight-gradient
    GEMMs are then complete).  ``clear_slots=False`` skips the second barrier and the zeroing of the
    consumed slots (for callers that overwrite, not accumulate into, the slots they use next time)."""
    lib = _native.load()
    n = len(states)
    args = (GradReduceArgs * n)()
    for i in range(n):
        a = GradReduceArgs()
        a.etc = ptr(etc_list[i])
        a.flags = (1 if entry_barrier else 0) | (4 if clear_slots else 2)
        pairs = tensor_pairs_list[i]
        a.ntensors = len(pairs)
        for j, (local, pool) in enumerate(pairs):
            a.t[j].local = local.data_ptr()
            a.t[j].pool = pool.data_ptr()
            a.t[j].expert_elems = local[0].numel()
            a.t[j].rank_stride = _rank_stride_bytes(pool)
        args[i] = a
    g = states[0].geo
    _native.check(lib.mep_launch_grad_reduce(n, _pack(states), args, g.num_sms, g.R, g.epn, _native.cur_stream()), "grad_reduce")
    if clear_slots:     # behind the kernel's second barrier, on all SMs (the cooperative kernel's few CTAs store slowly)
        sms = torch.cuda.get_device_properties(states[0].device).multi_processor_count
        _native.check(lib.mep_launch_grad_clear(n, _pack(states), args, 2 * sms, _native.cur_stream()), "grad_clear")


def launch_push_reduce(states, outs, out_ws, num_blocks):
    """Entry barrier + local sum over k of the rows the GEMM epilogues pushed into each rank's
    receive area (push-combine)."""
    lib = _native.load()
    n = len(states)
    args = (PushReduceArgs * n)()
    g = states[0].geo
    assert g.off_push, "this Buffer was created without the push-combine regions"
    for i in range(n):
        args[i] = PushReduceArgs(ptr(outs[i]), ptr(out_ws[i]) if out_ws is not None else None, g.off_push, g.off_pushw)
    _native.check(lib.mep_launch_push_reduce(n, _pack(states), args, num_blocks, _native.cur_stream()), "push_reduce")


def launch_wait_probe(st: RankState, flag: torch.Tensor, expected: int):
    lib = _native.load()
    _native.check(lib.mep_launch_wait_probe(C.c_void_p(st.ctx_ptr), C.c_void_p(flag.data_ptr()),
                                            C.c_uint32(expected), _native.cur_stream()), "wait_probe")
