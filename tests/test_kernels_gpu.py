"""Each fused sm_100a GEMM mode on its own against the plain torch implementation of the same op.

Follows the reference's kernel tests (tests/test_fused_kernels.py:18-67): forward intermediates `h`, `act`, `y` and
backward results `dx`, `dW_up`, `dW_down` one by one, bf16, tolerance 3e-2 of max-abs, group shapes with a partial
slice, an empty expert and a one-row expert; padding rows are poisoned with NaN and must not reach any result. Beyond
the reference's toy width the same checks run at real contraction depth (D=2048/F=1024, and D=7168/F=2048, the
DeepSeek-V3 expert), where a tile accumulates over 112 k-blocks.
"""

import math

import pytest
import torch

from chunked_ep_moe_b200.ops import expert as ref
from chunked_ep_moe_b200.ops import fused_expert as fx

pytestmark = pytest.mark.gpu

TOL = 3e-2

SHAPES = [
    # rows S, D, F, stripe, rows per expert
    (128, 256, 256, 128, [40, 0, 70]),      # partial slice (18 padding rows), empty expert
    (128, 256, 256, 64, [64, 1, 63]),       # full slice, one-row expert
    (512, 2048, 1024, 64, [130, 0, 255, 127]),
    (1024, 7168, 2048, 64, [300, 1, 270, 453]),
]


def _close(got, want, name, rows=None):
    got, want = got.float(), want.float()
    if rows is not None:
        got, want = got[:rows], want[:rows]
    assert torch.isfinite(got).all(), f"{name}: non-finite values"
    err = (got - want).abs().max() / want.abs().max().clamp_min(1e-6)
    assert err <= TOL, f"{name}: max abs err {err:.4f} x max-abs (allowed {TOL})"


def _inputs(S, D, F, groups, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    L, rows = len(groups), sum(groups)
    bf = torch.bfloat16
    x = torch.randn(S, D, generator=gen, device="cuda").to(bf)
    dy = torch.randn(S, D, generator=gen, device="cuda").to(bf)
    x[rows:] = float("nan")  # padding rows: whatever they hold must never matter
    dy[rows:] = float("nan")
    w_up = (torch.randn(L, D, 2 * F, generator=gen, device="cuda") / math.sqrt(D)).to(bf)
    w_down = (torch.randn(L, F, D, generator=gen, device="cuda") / math.sqrt(F)).to(bf)
    return x, dy, w_up, w_down, rows


@pytest.mark.parametrize("S,D,F,stripe,groups", SHAPES, ids=lambda v: str(v) if not isinstance(v, list) else "g")
def test_every_mode_matches_torch(S, D, F, stripe, groups):
    fx._runners.clear()
    x, dy, w_up, w_down, rows = _inputs(S, D, F, groups)
    sizes = torch.tensor(groups)

    # forward: act and h from the up-projection kernel, y from the plain grouped GEMM
    act, h = fx.gmm_swiglu(x, w_up, groups, stripe=stripe, return_h=True)
    want_h = ref.gmm(x, w_up, sizes, x.dtype)
    want_act = ref.striped_swiglu(want_h, stripe)
    _close(h, want_h, "h", rows)
    _close(act, want_act, "act", rows)
    y = fx.gmm(want_act, w_down, groups, stripe=stripe)
    _close(y, ref.gmm(want_act, w_down, sizes, x.dtype), "y", rows)
    act_only, none = fx.gmm_swiglu(x, w_up, groups, stripe=stripe)
    assert none is None
    _close(act_only, want_act, "act (no h)", rows)

    # backward, every kernel fed with the torch intermediates so that one kernel's error cannot hide another's
    want_dh = ref.striped_swiglu_bwd(want_h, ref.gmm(dy, w_down, sizes, x.dtype, transpose_rhs=True), stripe)
    dh = fx.gmm_dswiglu(dy, w_down, want_h, groups, stripe=stripe)
    _close(dh, want_dh, "dh", rows)
    dx = fx.gmm(want_dh, w_up, groups, transpose_rhs=True, stripe=stripe)
    _close(dx, ref.gmm(want_dh, w_up, sizes, x.dtype, transpose_rhs=True), "dx", rows)
    poisoned_act = want_act.clone()
    poisoned_act[rows:] = float("nan")
    poisoned_dh = want_dh.clone()
    poisoned_dh[rows:] = float("nan")
    dw_down = fx.tgmm(poisoned_act, dy, groups, stripe=stripe)
    _close(dw_down, ref.tgmm(want_act[:rows], dy[:rows], sizes), "dW_down")
    dw_up = fx.tgmm(x, poisoned_dh, groups, stripe=stripe)
    _close(dw_up, ref.tgmm(x[:rows], want_dh[:rows], sizes), "dW_up")
    for l, n in enumerate(groups):
        if n == 0:
            assert float(dw_up[l].abs().max()) == 0.0 and float(dw_down[l].abs().max()) == 0.0
    fx.check_status()


@pytest.mark.parametrize("S,D,F,stripe,groups", SHAPES[:3], ids=lambda v: str(v) if not isinstance(v, list) else "g")
def test_expert_forward_backward_wrappers(S, D, F, stripe, groups):
    """`expert_forward` / `expert_backward` (residual-consuming, nothing recomputed) against the torch pair."""
    fx._runners.clear()
    x, dy, w_up, w_down, rows = _inputs(S, D, F, groups, seed=3)
    sizes = torch.tensor(groups)
    y, res = fx.expert_forward(x, w_up, w_down, groups, stripe=stripe)
    want_y, want_res = ref.expert_forward(x[:rows], w_up, w_down, sizes, stripe=stripe)
    _close(y, want_y, "y", rows)
    _close(res.h, want_res.h, "h", rows)
    _close(res.act, want_res.act, "act", rows)
    grads = fx.expert_backward(x, w_up, w_down, groups, res, dy, stripe=stripe)
    want = ref.expert_backward(x[:rows], w_up, w_down, sizes, want_res, dy[:rows], stripe=stripe)
    _close(grads.dx, want.dx, "dx", rows)
    _close(grads.dw_up, want.dw_up, "dW_up")
    _close(grads.dw_down, want.dw_down, "dW_down")
    y_only, none = fx.expert_forward(x, w_up, w_down, groups, stripe=stripe, need_residuals=False)
    assert none is None
    _close(y_only, want_y, "y (no residuals)", rows)
    fx.check_status()


@pytest.mark.parametrize("groups", [[0, 0, 0], [0, 1, 0], [40, 0, 87], [64, 1, 63], [500, 7, 2]], ids=str)
def test_rows_past_the_groups_are_zero(groups):
    """The kernels write their outputs' padding rows themselves: none, all, and counts around the grid's CTAs."""
    S, D, F = (128 if sum(groups) <= 128 else 1024), 256, 512
    x, dy, w_up, w_down, rows = _inputs(S, D, F, groups)
    junk = [torch.full((S, 2 * F), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(8)]
    del junk  # the outputs are likely to land on these
    y, res = fx.expert_forward(x, w_up, w_down, groups, stripe=64)
    dh = fx.gmm_dswiglu(dy, w_down, res.h, groups, stripe=64)
    grads = fx.expert_backward(x, w_up, w_down, groups, res, dy, stripe=64)
    for name, t in (("y", y), ("h", res.h), ("act", res.act), ("dh", dh), ("dx", grads.dx)):
        assert torch.count_nonzero(t[rows:]) == 0 and torch.isfinite(t).all(), name
    fx.check_status()


def test_slices_in_preparation_do_not_share_tables():
    """Two slices of one geometry prepared before either runs (two threads, two streams): each keeps its own groups."""
    S, D, F = 256, 256, 256
    x, _, w_up, _, _ = _inputs(S, D, F, [256, 0, 0])
    groups = [[100, 0, 90], [3, 200, 53]]
    prepared = [fx._prepare(x, 3, g, 64) for g in groups]
    for runner, g in zip(prepared, groups):
        act, h = fx._gmm_swiglu(runner, x, w_up, True)
        want = fx.gmm_swiglu(x, w_up, g, stripe=64, return_h=True)
        assert torch.equal(act, want[0]) and torch.equal(h, want[1])
    fx.check_status()


@pytest.mark.parametrize("groups", [[0], [0, 0, 0], [0, 1, 0], [40, 0, 87]], ids=str)
def test_gradients_of_experts_without_rows_are_zero(groups):
    """Also when no expert has any (a rank's trailing slices under a collective transport)."""
    S, D, F = 128, 256, 256
    x, dy, w_up, w_down, _ = _inputs(S, D, F, groups)
    _, res = fx.expert_forward(x, w_up, w_down, groups, stripe=64)
    for t in (w_up, w_down):
        junk = [torch.full_like(t, float("nan")) for _ in range(4)]
        del junk  # the gradients are likely to land on these
    grads = fx.expert_backward(x, w_up, w_down, groups, res, dy, stripe=64)
    for name, t in (("dw_up", grads.dw_up), ("dw_down", grads.dw_down)):
        for g, n in zip(t, groups):
            assert torch.isfinite(g).all() and (n > 0 or torch.count_nonzero(g) == 0), name
    fx.check_status()


def test_weight_gradients_of_many_small_experts():
    """Experts of up to 320 rows keep their rows' panel along a row of tiles: none, one and five k-blocks, around each k-block's end and just
    past what a panel holds, in turn with experts that hold too many. NaN in one expert's rows and past the last one stays there."""
    L, M, N = 80, 1280, 1536  # 30 tiles an expert
    rows = [0, 1, 15, 16, 63, 64, 65, 320, 128, 200, 256, 257, 319, 321, 700, 48]
    groups = [rows[i % len(rows)] for i in range(L)]
    S = -(-sum(groups) // 8) * 8 + 8
    assert S <= 320 * L and 30 * L >= 32 * 74
    gen = torch.Generator(device="cuda").manual_seed(3)
    lhs = torch.randn(S, M, generator=gen, device="cuda").bfloat16()
    rhs = torch.randn(S, N, generator=gen, device="cuda").bfloat16()
    starts = [sum(groups[:i]) for i in range(L)]
    poisoned = 23  # 320 rows
    lhs[starts[poisoned]:starts[poisoned] + groups[poisoned]] = float("nan")
    rhs[starts[poisoned] + 3] = float("inf")
    lhs[sum(groups):] = float("nan")
    rhs[sum(groups):] = float("nan")
    for _ in range(2):
        out = fx.tgmm(lhs, rhs, groups)
        for g in range(L):
            at = slice(starts[g], starts[g] + groups[g])
            if g == poisoned:
                assert torch.isnan(out[g]).all()
                continue
            want = lhs[at].float().T @ rhs[at].float()
            # rounded once to bf16: 2^-9 of the value; the fp32 sums of up to 700 products differ by far less
            assert torch.linalg.vector_norm(out[g].float() - want) <= 2.0**-8 * torch.linalg.vector_norm(want), g
    fx.check_status()


def test_tiles_in_the_order_of_their_experts():
    """Large weights: an expert's tiles (none, 1, 2, 12, 13, 25) go over its weight columns together, at most 12 at a time. Every mode has the
    bits of calls on pieces of one expert's rows that are too short for that order."""
    D, F, stripe = 4096, 2048, 64
    groups = [0, 1, 3072, 3073, 0, 6400, 31, 257]
    S, L = sum(groups) + 6, len(groups)
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, dy = [torch.randn(S, D, generator=gen, device="cuda").bfloat16() for _ in range(2)]
    w_up = (0.02 * torch.randn(L, D, 2 * F, generator=gen, device="cuda")).bfloat16()
    w_down = (0.02 * torch.randn(L, F, D, generator=gen, device="cuda")).bfloat16()

    def every_mode(x, dy, w_up, w_down, groups):
        act, h = fx.gmm_swiglu(x, w_up, groups, stripe=stripe, return_h=True)
        return [act, h, fx.gmm(act, w_down, groups, stripe=stripe), fx.gmm(h, w_up, groups, transpose_rhs=True, stripe=stripe),
                fx.gmm_dswiglu(dy, w_down, h, groups, stripe=stripe)]

    whole = every_mode(x, dy, w_up, w_down, groups)
    assert all(torch.count_nonzero(t[sum(groups):]) == 0 for t in whole)
    at = 0
    for g, n in enumerate(groups):
        for begin in range(0, n, 1024):
            rows = min(1024, n - begin)
            piece = slice(at + begin, at + begin + rows)
            xs, dys = [torch.nn.functional.pad(t[piece], (0, 0, 0, -rows % 8)) for t in (x, dy)]
            alone = every_mode(xs, dys, w_up[g:g + 1], w_down[g:g + 1], [rows])
            for name, a, b in zip(("act", "h", "y", "dx", "dh"), whole, alone):
                assert torch.equal(a[piece], b[:rows]), (name, g, begin)
        at += n
    fx.check_status()


def test_kernels_refuse_rows_at_odd_addresses():
    """h and w * act are read 16 bytes at a time beside the tensor maps, which refuse other addresses of the operands."""
    S, D, F = 64, 256, 256
    bf = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    shifted = lambda t: torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)
    x, h, w_up, w_down = bf(S, D), bf(S, 2 * F), bf(2, D, 2 * F), bf(2, F, D)
    for call in (lambda: fx.gmm_dswiglu(x, w_down, shifted(h), [30, 34], stripe=64),
                 lambda: fx.gmm_dswiglu(shifted(x), w_down, h, [30, 34], stripe=64),
                 lambda: fx.gmm_swiglu(shifted(x), w_up, [30, 34], stripe=64), lambda: fx.gmm(shifted(x), w_up, [30, 34])):
        with pytest.raises(RuntimeError, match="16 bytes|16-byte"):
            call()
    fx.check_status()
