"""The fused sm_100a expert kernels one at a time: `gmm`, `gmm_swiglu`, `gmm_dswiglu`, `tgmm`, and the per-slice
`expert_forward` / `expert_backward` built from them.

Same kernel-level surface as the reference's fused backend (src/chunked_moe/kernels/fused_expert.py:102-366): every
function takes an expert-major slice of at most S rows plus the rows per expert, runs ONE tcgen05 grouped-GEMM mode
of `csrc/gemm/` on it, and returns tensors the caller owns. Rows past `sum(group_sizes)` are padding:
they are never read into a weight gradient and their outputs are left as allocated (zeros here).

This is what `expert_compute="fused"` runs under a COLLECTIVE transport (`ragged_a2a`, `emulated` on a GPU): the
exchange delivers a slice, these kernels compute on it, and the residuals (`h`, `act`) of the forward are handed to
the backward, so nothing is recomputed. Inside the NVLink path the same modes run fused with the transport
(`ops/fused.py`). The kernel tests compare each function with `ops/expert.py`.
"""

from __future__ import annotations

import os
from typing import Optional

import numpy as np
import torch

from .. import _build
from ..config import B200_NUM_SMS
from .expert import ExpertGrads, ForwardResiduals

_runners: dict = {}


def _group_tensor(group_sizes, device) -> torch.Tensor:
    if isinstance(group_sizes, torch.Tensor):
        return group_sizes.to(device=device, dtype=torch.int32).contiguous()
    return torch.from_numpy(np.asarray(group_sizes, dtype=np.int32)).to(device, non_blocking=True)


def _runner(num_groups: int, rows: int, stripe: int, device: torch.device):
    """The cached launcher for slices of `rows` rows and `num_groups` experts."""
    key = (num_groups, rows, stripe, device.index)
    runner = _runners.get(key)
    if runner is None:
        ext = _build.load()
        runner = ext.KernelRunner(num_groups, rows, stripe, int(os.environ.get("CEM_GEMM_GRID", B200_NUM_SMS)))
        _runners[key] = runner
    return runner


def _prepare(rows_tensor: torch.Tensor, num_groups: int, group_sizes, stripe: int):
    """A launcher with the tile tables of this slice (its own: calls on other streams or threads do not touch them)."""
    if rows_tensor.shape[0] % 8:
        raise ValueError(f"the fused kernels need a multiple of 8 rows per slice, got {rows_tensor.shape[0]}")
    runner = _runner(num_groups, rows_tensor.shape[0], stripe, rows_tensor.device)
    return runner.with_groups(_group_tensor(group_sizes, rows_tensor.device))


def _rows(runner, like: torch.Tensor, cols: int) -> torch.Tensor:
    """An output of the runner's kernels: they write the groups' rows and set the rows past the last group to zero."""
    return torch.empty((like.shape[0], cols), dtype=like.dtype, device=like.device)


def _gmm(runner, lhs, rhs, transpose_rhs):
    out = _rows(runner, lhs, rhs.shape[1] if transpose_rhs else rhs.shape[2])
    runner.gmm(lhs.contiguous(), rhs.contiguous(), out, transpose_rhs)
    return out


def _gmm_swiglu(runner, x, w_up, return_h):
    act = _rows(runner, x, w_up.shape[2] // 2)
    h = _rows(runner, x, w_up.shape[2]) if return_h else None
    runner.gmm_swiglu(x.contiguous(), w_up.contiguous(), act, h)
    return act, h


def _gmm_dswiglu(runner, dy, w_down, h):
    dh = _rows(runner, h, h.shape[1])
    runner.gmm_dswiglu(dy.contiguous(), w_down.contiguous(), h.contiguous(), dh)
    return dh


def _tgmm(runner, lhs, rhs, num_groups):
    out = lhs.new_empty((num_groups, lhs.shape[1], rhs.shape[1]))
    runner.tgmm(lhs.contiguous(), rhs.contiguous(), out)
    return out


def gmm(lhs: torch.Tensor, rhs: torch.Tensor, group_sizes, *, transpose_rhs: bool = False,
        stripe: int = 64) -> torch.Tensor:
    """`out[rows_g] = lhs[rows_g] @ rhs[g]` (`rhs [L, K, N]`), or `@ rhs[g]^T` (`rhs [L, N, K]`) with `transpose_rhs`."""
    return _gmm(_prepare(lhs, rhs.shape[0], group_sizes, stripe), lhs, rhs, transpose_rhs)


def gmm_swiglu(x: torch.Tensor, w_up: torch.Tensor, group_sizes, *, stripe: int,
               return_h: bool = False) -> tuple[torch.Tensor, Optional[torch.Tensor]]:
    """`act = silu(x Wg) * (x Wu)` from the striped `w_up [L, D, 2F]`; with `return_h` also the rounded `h [S, 2F]`."""
    return _gmm_swiglu(_prepare(x, w_up.shape[0], group_sizes, stripe), x, w_up, return_h)


def gmm_dswiglu(dy: torch.Tensor, w_down: torch.Tensor, h: torch.Tensor, group_sizes, *, stripe: int) -> torch.Tensor:
    """`dh = SwiGLU'(h) * (dy @ w_down[g]^T)`: the gradient of the striped pre-activation; `d_act` never leaves the SM."""
    return _gmm_dswiglu(_prepare(dy, w_down.shape[0], group_sizes, stripe), dy, w_down, h)


def tgmm(lhs: torch.Tensor, rhs: torch.Tensor, group_sizes, *, stripe: int = 64) -> torch.Tensor:
    """`out[g] = lhs[rows_g]^T @ rhs[rows_g]` -> `[L, lhs_cols, rhs_cols]` (bf16; fp32 accumulation over the rows)."""
    return _tgmm(_prepare(lhs, len(group_sizes), group_sizes, stripe), lhs, rhs, len(group_sizes))


def expert_forward(x: torch.Tensor, w_up: torch.Tensor, w_down: torch.Tensor, group_sizes, *, stripe: int,
                   need_residuals: bool = True) -> tuple[torch.Tensor, Optional[ForwardResiduals]]:
    runner = _prepare(x, w_up.shape[0], group_sizes, stripe)  # one build of the tile tables for the call's kernels
    act, h = _gmm_swiglu(runner, x, w_up, need_residuals)
    y = _gmm(runner, act, w_down, False)
    return y, (ForwardResiduals(h=h, act=act) if need_residuals else None)


def expert_backward(x: torch.Tensor, w_up: torch.Tensor, w_down: torch.Tensor, group_sizes, res: ForwardResiduals,
                    dy: torch.Tensor, *, stripe: int) -> ExpertGrads:
    groups = w_up.shape[0]
    runner = _prepare(dy, groups, group_sizes, stripe)
    dh = _gmm_dswiglu(runner, dy, w_down, res.h)
    return ExpertGrads(dx=_gmm(runner, dh, w_up, True), dw_up=_tgmm(runner, x, dh, groups),
                       dw_down=_tgmm(runner, res.act, dy, groups))


def check_status() -> None:
    """Synchronises and raises if a kernel launched through this module recorded an error."""
    for runner in _runners.values():
        runner.check_status()
