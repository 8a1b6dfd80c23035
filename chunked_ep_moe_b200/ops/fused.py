"""The fused NVLink path: `chunked_moe` on the sm_100a kernels (`transport="nvshmem"`, `expert_compute="fused"`).

Per pass the host launches, per slice, a put kernel on the comm stream and a handful of grouped
tcgen05 GEMMs on the compute streams; everything between ranks happens inside those kernels
(peer stores, arrival counters, credits). The host never waits for the device inside a pass: the
slice count of a forward is guessed from the previous pass and corrected once its real value has
reached the host. Compared with the reference's loop
(src/chunked_moe/moe.py:96-119, :148-206):

  * no `[T*K, D]` send buffer: the put kernel gathers rows straight from `x[token]`;
  * the router weight is applied in the up-projection epilogue (`w * act`); the down-projection's stores every finished
    row into the source rank's return buffer; a local K-way fixed-order sum finishes the token;
  * `d_weight = <g, act Wd>` is `<g Wd^T, act>`, a by-product of the GEMM that yields `d_act = w * (g Wd^T)`, and
    `dW_down` contracts `w * act` with `g`; neither `y` nor `w * g` exists;
  * the backward starts from `h` and `w * act` where the forward could keep them (large slices, memory to spare,
    `CEM_KEEP_ACTIVATIONS=0` never) and recomputes them, slice by slice, where it could not: the same bits either way;
  * weight gradients are written once per expert in bf16; only the (at most one) expert that
    straddles a slice boundary carries an fp32 partial to the next slice;
  * a rank on its own exchanges nothing, so its passes run as ONE slice, in up to eight ranges of experts, as long as their
    buffers fit beside what is live in half of the device's memory (`FusedRank::runs_whole`); slice by slice otherwise, with
    `always_slice` and under saved-tensor hooks. Passes of one range also keep x in expert order, as long as live tensors stay within a
    quarter of the device; forwards of few tokens gather their rows in the up-projection (`FusedRank::runs_brief`).

Everything else the backward needs are the inputs and the integer plan (tables, send order, its inverse).
"""

from __future__ import annotations

import contextlib
import math
import os
import threading
from typing import Optional

import torch
import torch.distributed as dist

from .. import _build
from ..config import ChunkedMoEConfig
from ..parallel.symm import SymmetricArena

_DEFAULT_SPIN_LIMIT = 1 << 24  # polls (~0.3 us each) before a wait on another rank gives up
_PUT_BLOCKS = 128  # measured: 128 blocks finish a put soonest and disturb the GEMM beside it least

_workspaces: dict = {}
_retired: list = []  # workspaces replaced by `reserve()`; passes in flight may still hold them
_making: dict = {}  # a lock for every geometry and group whose workspace is being made or replaced

#: Pass as `group` to run the fused kernels on this rank alone (a 1-rank expert-parallel world), whatever
#: process groups exist. Used by `ops.fused_expert` to serve `expert_compute="fused"` on collective transports.
SOLO = "solo"


class FusedWorkspace:
    """Symmetric arena + per-rank executor for one (geometry, process group)."""

    def __init__(self, cfg: ChunkedMoEConfig, group, hidden: int, ffn: int, tk_cap: int):
        ext = _build.load()
        initialised = dist.is_available() and dist.is_initialized() and group is not SOLO
        self.world = dist.get_world_size(group) if initialised else 1
        self.rank_index = dist.get_rank(group) if initialised else 0
        self.local_experts = cfg.num_experts // self.world
        if group is SOLO:
            group = None
        if self.world > 1:  # the arena layout must be identical everywhere: agree on the capacity
            cap = torch.tensor([tk_cap], device="cuda", dtype=torch.int64)
            dist.all_reduce(cap, op=dist.ReduceOp.MAX, group=group)
            tk_cap = int(cap.item())
        self.tk_cap = tk_cap
        self.fp8 = cfg.comm_dtype == "float8_e4m3fn"
        self.max_slices = max(1, math.ceil(self.world * tk_cap / cfg.slice_size)) + 1
        nbytes = ext.arena_bytes(self.world, self.local_experts, cfg.slice_size, hidden, tk_cap, self.fp8)
        self.arena = SymmetricArena(nbytes, group, solo=self.world == 1)
        self.rank = ext.FusedRank(
            P=self.world, L=self.local_experts, me=self.rank_index, S=cfg.slice_size, D=hidden, F=ffn, K=cfg.top_k,
            stripe=cfg.stripe_width, tk_cap=tk_cap, max_slices=self.max_slices,
            num_sms=int(os.environ.get("CEM_GEMM_GRID", cfg.num_sms)), fp8=self.fp8,
            arena=self.arena.local, peer_arenas=self.arena.peers, use_comm_stream=True,
            spin_limit=int(os.environ.get("CEM_SPIN_LIMIT", _DEFAULT_SPIN_LIMIT)),
            put_blocks=int(os.environ.get("CEM_PUT_BLOCKS", _PUT_BLOCKS)))
        self.rank.set_whole_passes(not cfg.always_slice)
        if "CEM_MBAR_LIMIT_US" in os.environ:
            self.rank.set_mbar_limit_us(int(os.environ["CEM_MBAR_LIMIT_US"]))
        self.plan_ints = self.rank.plan_ints()
        self.dummy_counts = torch.zeros(1, dtype=torch.int32, device="cuda")


def _workspace_key(cfg: ChunkedMoEConfig, group, hidden: int, ffn: int):
    # The process group OBJECT is part of the key (not its id): the dictionary keeps it alive, so a later group can
    # never be mistaken for it.
    return (group, cfg.num_experts, cfg.top_k, cfg.slice_size, cfg.stripe_width, cfg.comm_dtype, cfg.num_sms,
            cfg.always_slice, hidden, ffn, torch.cuda.current_device())


@contextlib.contextmanager
def _alone_with(key):
    """One thread at a time makes or replaces a geometry's workspace. (No lock for all of them: making one is collective, and the threads
    of two ranks may come to two groups in different orders.)"""
    while True:
        lock = _making.setdefault(key, threading.Lock())
        with lock:
            if _making.get(key) is lock:  # (else whoever was waited for has taken it away)
                try:
                    yield
                finally:
                    del _making[key]  # the key holds a process group
                return


def get_workspace(cfg: ChunkedMoEConfig, group, hidden: int, ffn: int, tokens_times_k: int) -> FusedWorkspace:
    """The cached workspace for this geometry and group; the first call creates it (collectively).

    A workspace never shrinks, moves or is freed behind a pass that still holds it: its capacity is fixed when it is
    created (the largest `T*K` over the ranks at that moment). A later call that needs more gets a new, larger one
    when this rank is alone; among several ranks it raises, because making room is a collective decision:
    `reserve()` is the way to do that.
    """
    key = _workspace_key(cfg, group, hidden, ffn)
    ws = _workspaces.get(key)
    if ws is None:
        with _alone_with(key):
            ws = _workspaces.get(key)  # (another thread's by now?)
            if ws is None:
                ws = _workspaces[key] = FusedWorkspace(cfg, group, hidden, ffn, tokens_times_k)
    if ws.tk_cap >= tokens_times_k:
        return ws
    if ws.world == 1:
        return reserve(cfg, group, hidden, ffn, tokens_times_k)  # nobody to agree with: make room right away
    raise RuntimeError(
        f"chunked_moe fused path: this call has {tokens_times_k} token copies but the workspace of this geometry "
        f"was created for {ws.tk_cap}. Capacity is agreed between the ranks when the workspace is created; call "
        f"ops.fused.reserve(cfg, group, hidden, ffn, tokens_times_k) on every rank first.")


def reserve(cfg: ChunkedMoEConfig, group, hidden: int, ffn: int, tokens_times_k: int) -> FusedWorkspace:
    """Collective: makes sure the workspace of this geometry holds `tokens_times_k` token copies on every rank.

    A workspace that is too small is replaced, not freed: passes whose backward has not run yet keep using the arena
    they started with, and the old workspace is only released by `release_workspaces()`.
    """
    key = _workspace_key(cfg, group, hidden, ffn)
    with _alone_with(key):
        ws = _workspaces.get(key)
        need = tokens_times_k
        if dist.is_available() and dist.is_initialized() and group is not SOLO and dist.get_world_size(group) > 1:
            t = torch.tensor([need, ws.tk_cap if ws is not None else 0], device="cuda", dtype=torch.int64)
            dist.all_reduce(t, op=dist.ReduceOp.MAX, group=group)
            need, have = int(t[0]), int(t[1])
        else:
            have = ws.tk_cap if ws is not None else 0
        if ws is None or have < need:  # every rank takes the same branch: both numbers are maxima over the ranks
            if ws is not None:
                _retired.append(ws)
            ws = _workspaces[key] = FusedWorkspace(cfg, group, hidden, ffn, need)
        return ws


def release_workspaces() -> None:
    """Frees every workspace, cached or replaced (collective when a process group is involved). A pass whose backward
    has not run yet must not be kept across this call: its backward raises."""
    going = [ws for ws in (_workspaces.pop(key, None) for key in list(_workspaces)) if ws is not None]
    while _retired:
        going.append(_retired.pop(0))
    for ws in going:  # (what another thread makes meanwhile stays, for its next call)
        if ws.rank is not None:
            ws.rank.release()
        ws.rank = None
        ws.arena.close()


def _ranks() -> list:
    return [rank for rank in (ws.rank for ws in list(_workspaces.values())) if rank is not None]


def last_plan_stats(cfg: ChunkedMoEConfig) -> list:
    """Load statistics of the most recent pass of every cached workspace (rows, slices, padding, remote rows)."""
    from ..utils.stats import header_stats

    return [header_stats(list(rank.plan_header()), cfg.slice_size) for rank in _ranks()]


def check_status() -> None:
    """Synchronises and raises if any kernel of a cached workspace recorded an error (a wait that ran out).

    The forward checks on its own (it has to read the slice count back anyway); the backward does not synchronise,
    so a training loop calls this once per step, before the optimizer consumes the gradients.
    """
    for rank in _ranks():
        rank.check_status()


def launches() -> int:
    """Kernels launched so far by every cached workspace of this process."""
    return sum(int(rank.launches()) for rank in _ranks())


def expected_launches(num_slices: int, fp8: bool = False, kept_slices: int = 0) -> int:
    """Kernels one forward+backward of the fused layer launches on a rank that loops `num_slices` slices.

    Forward: sort (3) + plan build + pass begin + per slice (put, swiglu, down+combine, slice done) + combine reduce.
    Backward: pass begin + per slice (put, swiglu+h, dswiglu, dW_down, d_weight return, dx+combine, dW_up, slice done)
    + combine reduce. `fp8`: among several ranks the fp8 wire adds one expansion kernel per slice and pass (a rank on its own
    launches none: pass False). A slice whose activations the forward kept needs no swiglu+h in the backward. (A rank on its
    own loops slices with `always_slice`, under saved-tensor hooks or when memory is short; otherwise `expected_launches_alone`.)
    """
    per_slice = 12 + (2 if fp8 else 0)
    return 8 + per_slice * num_slices - kept_slices


def expected_launches_alone(rows: int, experts: int, hidden: int, ffn: int, kept: bool) -> int:
    """Kernels one forward+backward launches on a rank on its own that runs it as one slice; `kept`: h and w * act stay.

    Forward: sort and plan (3, or 1 up to 2048 ids and 512 experts) + per range of experts (put, swiglu, down+combine) + combine
    reduce. Backward: per range (put, dswiglu, dW_down, dx+combine, dW_up, and swiglu+h or, beside the first GEMM of several kept
    ranges, a put of x) + d_weight return + combine reduce. (A forward of one slice, up to 2048 ids and 512 experts, without
    autograd: 5, also with `always_slice`; otherwise up to 96 tokens 4, up to 32 ids 3.)
    """
    ext = _build.load()
    forward, backward = [ext.whole_ranges(rows, experts, hidden, ffn, True, b) for b in (False, True)]
    plan = 1 if rows <= ext.plan_small[0] and experts <= ext.plan_small[1] else 3
    return plan + 1 + 3 * forward + 2 + (5 if kept and backward == 1 else 6) * backward


def memory_plan(world: int, experts: int, top_k: int, tokens_per_rank: int, hidden: int, ffn: int, slice_size: int,
                fp8: bool = False, tk_cap: int | None = None, always_slice: bool = False) -> dict:
    """Bytes one rank of the fused path holds, by purpose (no GPU needed: sizes come from the arena layout).

    `tk_cap` is the workspace capacity in token copies (default `tokens_per_rank * top_k`).
    """
    ext = _build.load()
    L = experts // world
    alone = world == 1 and not always_slice  # passes run as one slice
    tk = tokens_per_rank * top_k if tk_cap is None else tk_cap
    S, D, F = slice_size, hidden, ffn
    arena = int(ext.arena_bytes(world, L, S, D, tk, fp8))
    scratch = 2 * (S * F * 2 + S * 2 * F * 2 + S * 2 * F * 2 + S * (F // 32) * 4)  # act, h, dh, d_weight shares, x2
    carry = 2 * (D * 2 * F + F * D) * 4
    weights = L * (D * 2 * F + F * D) * 2
    max_slices = max(1, math.ceil(world * tk / S)) + 1
    plan = int(ext.plan_layout(world, L, S, max_slices)["total"]) * 4
    saved = tokens_per_rank * D * 2 + tk * 4 * 3 + plan  # x, router weights, order, inverse order, plan tables
    out = {
        "arena (slice buffers x2 for x and g, return rows, counters, traffic matrix)": arena,
        "scratch (act, h, dh, d_weight shares; two slices in flight)": scratch,
        "weight-gradient carry tiles (fp32, two per matrix)": carry,
        "expert weights (bf16)": weights,
        "expert weight gradients (bf16)": weights,
        "saved for backward (x, router weights, sort order, plan)": saved,
        "kept for backward while memory allows (h, w * act; rows balanced over the ranks)":
            tk * 3 * F * 2 if (tk if alone else min(tk, S)) * D * F >= ext.keep_work else 0,
    }
    if alone:
        out["during a pass that runs as one slice, while memory allows (x, g, dh by rows; x up to the backward, while a quarter of the "
            "device allows)"] = tk * (2 * D + 2 * F) * 2
    out["total"] = sum(out.values())
    return out


PIPELINE_COUNTER_SLOTS = ("loop_cycles", "loop_ns", "producer_wait_free_stage", "mma_wait_filled_stage",
                          "mma_wait_accumulator", "k_blocks", "epilogue_wait_accumulator", "tiles")
GEMM_MODE_NAMES = ("swiglu", "down_fwd", "unused", "dswiglu", "dx", "tgmm")


def pipeline_counters(enable: bool = True) -> list:
    """Turns the GEMM kernels' in-kernel pipeline counters on (or off) for every cached workspace.

    Returns one zeroed int64 tensor `[6 modes, CTAs, 8 slots]` per workspace (slot names:
    `PIPELINE_COUNTER_SLOTS`); every later GEMM launch adds its CTAs' cycle counts to it. The counters say which
    side of the operand ring waits for the other (loads or MMAs) and, from cycles / nanoseconds, the SM clock the
    kernels really ran at. Diagnostics: counting costs a few clock reads per k-block.
    """
    out = []
    for rank in _ranks():
        if not enable:
            rank.set_pipeline_counters(None)
            continue
        t = torch.zeros(6, max(148, torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count),
                        len(PIPELINE_COUNTER_SLOTS), dtype=torch.int64, device="cuda")
        rank.set_pipeline_counters(t)
        out.append(t)
    return out


def _require(cond: bool, msg: str) -> None:
    if not cond:
        raise ValueError("chunked_moe fused path: " + msg)


def unsupported_reason(x: torch.Tensor, w_up: torch.Tensor, w_down: torch.Tensor,
                       cfg: ChunkedMoEConfig) -> Optional[str]:
    """Why these tensors cannot run on the fused kernels (shape or dtype), or None. The caller may then fall back to
    a collective transport, as the reference's put kernel does for rows it cannot move
    (src/chunked_moe/transport/nvshmem.py:115-118)."""
    if x.dtype != torch.bfloat16 or w_up.dtype != torch.bfloat16 or w_down.dtype != torch.bfloat16:
        return "x, w_up and w_down must be bfloat16"
    if x.shape[1] % 256 or w_down.shape[1] % 256:
        return f"D={x.shape[1]} and F={w_down.shape[1]} must be multiples of 256"
    if cfg.stripe_width not in (32, 64, 128):
        return f"stripe_width={cfg.stripe_width} must be 32, 64 or 128"
    if cfg.slice_size % 8:
        return f"slice_size={cfg.slice_size} must be a multiple of 8"
    if cfg.accum_dtype != "float32":
        return f"accum_dtype={cfg.accum_dtype!r}: the kernels accumulate weight gradients in float32"
    return None


def chunked_moe_fused(x: torch.Tensor, expert_ids: torch.Tensor, weights: torch.Tensor, w_up: torch.Tensor,
                      w_down: torch.Tensor, cfg: ChunkedMoEConfig,
                      group: Optional[dist.ProcessGroup] = None) -> torch.Tensor:
    _require(cfg.expert_compute == "fused", 'transport="nvshmem" requires expert_compute="fused"')
    _require(x.is_cuda, "inputs must be CUDA tensors (the sm_100a extension has no CPU path)")
    _require(x.dtype == torch.bfloat16 and w_up.dtype == torch.bfloat16 and w_down.dtype == torch.bfloat16,
             "x, w_up and w_down must be bfloat16")
    _require(x.shape[1] % 256 == 0 and w_down.shape[1] % 256 == 0, "needs D % 256 == 0 and F % 256 == 0")
    _require(cfg.stripe_width in (32, 64, 128), "needs stripe_width in {32, 64, 128}")
    _require(cfg.slice_size % 8 == 0, "needs slice_size % 8 == 0")
    _require(cfg.accum_dtype == "float32", "weight gradients are accumulated in float32 (accum_dtype)")
    tokens, hidden = x.shape
    ws = get_workspace(cfg, group, hidden, w_down.shape[1], tokens * cfg.top_k)
    return _build.load().chunked_moe_layer(ws.rank, x, expert_ids, weights, w_up, w_down)
