"""The decoder's fused CUDA ops (residual add + RMSNorm, rotary embedding out of qkv, cross-entropy of bf16 logits, router)
against plain PyTorch fp32 references of the same ops, forward and backward."""

import math

import pytest
import torch
import torch.nn.functional as F

from chunked_ep_moe_b200.models import fused_ops

pytestmark = pytest.mark.gpu


def _close(got, want, name, tol):
    got, want = got.float(), want.float()
    assert torch.isfinite(got).all(), f"{name}: non-finite values"
    err = (got - want).abs().max() / want.abs().max().clamp_min(1e-6)
    assert err <= tol, f"{name}: max abs err {err:.5f} x max-abs (allowed {tol})"


@pytest.mark.parametrize("rows,cols,with_delta", [(300, 1024, True), (64, 2048, True), (129, 256, False)])
def test_add_rms_norm(rows, cols, with_delta):
    gen = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(rows, cols, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    delta = torch.randn(rows, cols, device="cuda", generator=gen).bfloat16().requires_grad_(True) if with_delta else None
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=gen)).bfloat16().requires_grad_(True)
    gs = torch.randn(rows, cols, device="cuda", generator=gen).bfloat16()
    gy = torch.randn(rows, cols, device="cuda", generator=gen).bfloat16()
    s, y = fused_ops.add_rms_norm(x, delta, w, 1e-6)
    (s.float() * gs.float()).sum().add((y.float() * gy.float()).sum()).backward()
    xr = x.detach().float().requires_grad_(True)
    dr = delta.detach().float().requires_grad_(True) if with_delta else None
    wr = w.detach().float().requires_grad_(True)
    sr = xr
    if with_delta:  # the sum is stored rounded to bf16; gradients pass straight through the rounding
        sr = xr + dr + ((xr + dr).detach().bfloat16().float() - (xr + dr).detach())
    yr = sr * torch.rsqrt(sr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    (sr * gs.float()).sum().add((yr * gy.float()).sum()).backward()
    _close(s, sr.detach(), "s", 1e-2)
    _close(y, yr.detach(), "y", 1e-2)
    _close(x.grad, xr.grad, "dx", 2e-2)
    if with_delta:
        _close(delta.grad, dr.grad, "ddelta", 2e-2)
    _close(w.grad, wr.grad, "dweight", 2e-2)


def test_rope_qkv():
    B, S, H, hd = 2, 96, 4, 64
    gen = torch.Generator(device="cuda").manual_seed(1)
    qkv = torch.randn(B, S, 3, H, hd, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    inv = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, device="cuda", dtype=torch.float32) / hd))
    ang = torch.outer(torch.arange(S, device="cuda", dtype=torch.float32), inv)
    cos, sin = ang.cos(), ang.sin()
    g = [torch.randn(B, H, S, hd, device="cuda", generator=gen).bfloat16() for _ in range(3)]
    q, k, v = fused_ops.rope_qkv(qkv, cos, sin)
    sum((t.float() * gi.float()).sum() for t, gi in zip((q, k, v), g)).backward()

    ref = qkv.detach().float().requires_grad_(True)
    rq, rk, rv = ref.permute(2, 0, 3, 1, 4)

    def rot(x):
        xc = torch.view_as_complex(x.reshape(*x.shape[:-1], -1, 2).contiguous())
        return torch.view_as_real(xc * torch.complex(cos, sin)).flatten(-2)

    outs = (rot(rq), rot(rk), rv)
    sum((t * gi.float()).sum() for t, gi in zip(outs, g)).backward()
    for name, a, b in zip("qkv", (q, k, v), outs):
        _close(a, b.detach(), name, 1e-2)
    _close(qkv.grad, ref.grad, "dqkv", 1e-2)


@pytest.mark.parametrize("rows,cols", [(257, 32000), (16, 1024)])
def test_cross_entropy(rows, cols):
    gen = torch.Generator(device="cuda").manual_seed(2)
    logits = (3 * torch.randn(rows, cols, device="cuda", generator=gen)).bfloat16().requires_grad_(True)
    targets = torch.randint(0, cols, (rows,), device="cuda", generator=gen)
    loss = fused_ops.cross_entropy(logits, targets)
    (loss * 1.7).backward()
    ref = logits.detach().float().requires_grad_(True)
    want = F.cross_entropy(ref, targets)
    (want * 1.7).backward()
    assert abs(float(loss) - float(want)) <= 1e-3 * max(1.0, abs(float(want)))
    _close(logits.grad, ref.grad, "dlogits", 1e-2)


@pytest.mark.parametrize("cols", [8, 2040, 2048, 2056, 8184, 8192, 8200, 10248])
def test_cross_entropy_row_widths(cols):
    """A thread's loads of a row full, partly and just filled; rows that begin with masked logits, have one in sight, have an infinity or a
    NaN. The log-sum-exp is fp32 sums of positive terms: 2^-24 for each of the at most 8 + 13 additions and 4 roundings on a term's way,
    and of the result."""
    gen = torch.Generator(device="cuda").manual_seed(cols)
    logits = (4 * torch.randn(9, cols, device="cuda", generator=gen)).bfloat16()
    logits[0, : cols - 1] = -float("inf")
    logits[1, : cols // 2] = -float("inf")
    logits[2, cols // 2] = float("nan")
    logits[3, cols // 2] = float("inf")
    logits[4] = -1e30
    targets = torch.full((9,), cols - 1, device="cuda")
    loss, lse = fused_ops._ext().cross_entropy_fwd(logits, targets)
    want = torch.logsumexp(logits.double(), 1)
    assert torch.isnan(lse[2]) and not torch.isfinite(loss[3])
    rest = [0, 1, 4, 5, 6, 7, 8]
    assert ((lse.double() - want).abs() <= (64 + want.abs()) * 2.0**-24)[rest].all()
    torch.testing.assert_close(loss[rest], (want - logits[:, -1].double())[rest].float(), rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("tokens,experts,top_k", [(1, 32, 32), (700, 64, 6), (5000, 256, 8)])
def test_router_select_of_equal_and_negative_scores(tokens, experts, top_k):
    """Ties go to the lower expert, zeros of either sign are equal, and the order holds below zero; the counts are those of the ids."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    logits = torch.randint(-2, 3, (tokens, experts), generator=gen, device="cuda").float()
    bias = torch.randint(-3, 1, (experts,), generator=gen, device="cuda").float()
    logits[0] = float("-inf")  # scores of 0
    bias[::2], bias[1::3] = 0.0, -0.0
    ids, _, counts, _ = fused_ops.router_select(logits, bias, top_k, 1.0)
    keys = 1.0 / (1.0 + torch.exp(-logits)) + bias
    order = torch.sort(keys, dim=1, descending=True, stable=True).indices[:, :top_k]
    picked, best = torch.gather(keys, 1, ids.long()), torch.gather(keys, 1, order)
    assert torch.equal(ids[0].long(), order[0])
    # (exp and the kernel's differ in the last bits, so that sums which are equal in one may not be in the other)
    assert (picked - best).abs().max() <= 1e-6
    assert (torch.sort(ids.long(), dim=1).values.diff(dim=1) > 0).all()
    assert torch.equal(counts.long(), torch.bincount(ids.long().reshape(-1), minlength=experts))


@pytest.mark.parametrize("tokens,experts,top_k", [(1000, 64, 6), (8192, 256, 8), (7, 32, 1), (333, 96, 5)])
def test_router_select(tokens, experts, top_k):
    """Selection, weights, load counts, score sums and the gradient w.r.t. the logits against fp64 torch ops."""
    gen = torch.Generator(device="cuda").manual_seed(tokens + experts)
    logits = torch.randn(tokens, experts, generator=gen, device="cuda").requires_grad_(True)
    bias = 0.1 * torch.randn(experts, generator=gen, device="cuda")
    gw = torch.randn(tokens, top_k, generator=gen, device="cuda")
    gs = torch.randn(experts, generator=gen, device="cuda")
    scaling = 2.5
    ids, weights, counts, sums = fused_ops.router_select(logits, bias, top_k, scaling)
    ((weights * gw).sum() + (sums * gs).sum()).backward()
    assert ids.dtype == torch.int32 and tuple(ids.shape) == (tokens, top_k)

    ref_logits = logits.detach().double().requires_grad_(True)
    scores = torch.sigmoid(ref_logits)
    keys = (scores + bias.double()).detach()
    picked = torch.gather(keys, 1, ids.long())
    # a valid top-k: distinct experts, in descending order of score + bias, none of the others beats the last one
    assert (torch.sort(ids.long(), dim=1).values.diff(dim=1) > 0).all() or top_k == 1
    assert (picked.diff(dim=1) <= 1e-6).all()
    rest = keys.scatter(1, ids.long(), float("-inf"))
    assert (rest.max(dim=1).values <= picked[:, -1] + 1e-6).all()
    chosen = torch.gather(scores, 1, ids.long())
    ref_weights = chosen / chosen.sum(-1, keepdim=True).clamp_min(1e-20) * scaling
    ref_sums = (scores / scores.sum(-1, keepdim=True).clamp_min(1e-20)).sum(0)
    ((ref_weights * gw.double()).sum() + (ref_sums * gs.double()).sum()).backward()
    torch.testing.assert_close(weights.double(), ref_weights.detach(), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(counts.long(), torch.bincount(ids.long().reshape(-1), minlength=experts))
    torch.testing.assert_close(sums.double(), ref_sums.detach(), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(logits.grad.double(), ref_logits.grad, rtol=1e-4, atol=1e-6)


def test_router_select_is_deterministic():
    gen = torch.Generator(device="cuda").manual_seed(5)
    logits = torch.randn(4096, 64, generator=gen, device="cuda")
    bias = torch.zeros(64, device="cuda")
    a = fused_ops.router_select(logits, bias, 6, 1.0)
    b = fused_ops.router_select(logits, bias, 6, 1.0)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("rows,ffn", [(300, 512), (8192, 2048), (5, 8)])
def test_dense_swiglu(rows, ffn):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    gu = torch.randn(rows, 2 * ffn, device="cuda", generator=gen).bfloat16().requires_grad_(True)
    go = torch.randn(rows, ffn, device="cuda", generator=gen).bfloat16()
    out = fused_ops.dense_swiglu(gu)
    out.backward(go)
    ref_in = gu.detach().float().requires_grad_(True)
    gate, up = ref_in.chunk(2, dim=-1)
    ref = F.silu(gate) * up
    ref.backward(go.float())
    _close(out, ref, "act", 1e-2)
    _close(gu.grad, ref_in.grad, "d_gate_up", 1e-2)


@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 248), (9, 256), (33, 264), (8, 768), (2369, 776), (5, 1032), (2, 2040)])
def test_add_rms_norm_row_widths(rows, cols):
    """Every number of 16-byte units per lane, with ragged last units, and more rows than the grid has warps."""
    gen = torch.Generator(device="cuda").manual_seed(cols)
    x, delta, gs, gy = [torch.randn(rows, cols, device="cuda", generator=gen).bfloat16() for _ in range(4)]
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=gen)).bfloat16()
    leaves = [t.clone().requires_grad_(True) for t in (x, delta, w)]
    s, y = fused_ops.add_rms_norm(*leaves, 1e-6)
    torch.autograd.backward([s, y], [gs, gy])
    sr = (x.float() + delta.float()).bfloat16().double().requires_grad_(True)
    wr = w.double().requires_grad_(True)
    yr = sr * torch.rsqrt(sr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    torch.autograd.backward([sr, yr], [gs.double(), gy.double()])
    assert torch.equal(s.double(), sr.detach())
    # one rounding to bf16 (2^-9 of the value) on top of fp32 arithmetic
    for name, got, want in (("y", y, yr.detach()), ("dx", leaves[0].grad, sr.grad), ("dw", leaves[2].grad, wr.grad)):
        assert (got.double() - want).abs().le(want.abs() * 2.0**-8 + 1e-5 * want.abs().max()).all(), name
    assert torch.equal(leaves[0].grad, leaves[1].grad)


@pytest.mark.parametrize("tokens,vocab,cols", [(1, 1, 8), (31, 7, 8), (33, 256, 264), (1025, 257, 256), (16384, 40, 264),
                                               (16384, 1, 8), (500, 1 << 18, 8), (8191, 32000, 1032)])
def test_embedding_gradient(tokens, vocab, cols):
    """Rows with no, few and many pairs, one to three digits of the ids, ragged columns. fp32 sums of n terms (n 2^-24 of the sum
    of their magnitudes) and one rounding to bf16 (2^-9 of the value; twice both allowed). The same bits every time."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    ids = torch.randint(0, vocab, (1, tokens), generator=gen, device="cuda")
    ids[0, tokens // 2:] = ids[0, tokens // 2:] // 3  # unevenly
    g = torch.randn(1, tokens, cols, generator=gen, device="cuda").bfloat16()
    grads = []
    for _ in range(2):
        weight = torch.randn(vocab, cols, generator=gen, device="cuda").bfloat16().requires_grad_(True)
        out = fused_ops.embedding(ids, weight)
        assert torch.equal(out, F.embedding(ids, weight))
        out.backward(g)
        grads.append(weight.grad)
    sums = lambda t: torch.zeros(vocab, cols, device="cuda", dtype=torch.float64).index_add_(0, ids[0], t)
    want, size = sums(g[0].double()), sums(g[0].double().abs())
    count = torch.bincount(ids[0], minlength=vocab)[:, None]
    assert (grads[0].double() - want).abs().le(2.0**-8 * want.abs() + count * 2.0**-23 * size).all()
    assert torch.equal(*grads)


@pytest.mark.parametrize("cols", [8, 40, 520])
def test_embedding_gradient_of_rows_with_many_pairs(cols):
    """Rows of 0, 1, 15, 16, 17, ... pairs: around the 16 up to which one warp sums a row, the 512 that 64 lane groups have in flight,
    and a row of most of the pairs. Bounds as above; the same bits every time."""
    counts = torch.tensor([0, 1, 15, 16, 17, 31, 32, 33, 0, 63, 64, 65, 511, 512, 513, 1025, 4097, 3], device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(cols)
    ids = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), counts)
    ids = ids[torch.randperm(len(ids), generator=gen, device="cuda")]
    g = torch.randn(len(ids), cols, generator=gen, device="cuda").bfloat16()
    grads = []
    for _ in range(2):
        weight = torch.zeros(len(counts), cols, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        fused_ops.embedding(ids, weight).backward(g)
        grads.append(weight.grad)
    sums = lambda t: torch.zeros(len(counts), cols, device="cuda", dtype=torch.float64).index_add_(0, ids, t)
    want, size = sums(g.double()), sums(g.double().abs())
    assert (grads[0].double() - want).abs().le(2.0**-8 * want.abs() + counts[:, None] * 2.0**-23 * size).all()
    assert torch.equal(*grads)


@pytest.mark.parametrize("ids", ["zipf", "padded"])
@pytest.mark.parametrize("tokens,cols", [(8192, 1024), (16384, 2048)])
def test_embedding_gradient_of_skewed_ids_is_no_slower_than_the_frameworks(tokens, cols, ids):
    """Ids of text (the commonest word 9 % of them) and of a batch that is mostly padding: one row of the table has many pairs."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    if ids == "zipf":
        popularity = 1.0 / torch.arange(1, 32001, device="cuda", dtype=torch.float32)
        tok = torch.multinomial(popularity, tokens, replacement=True, generator=gen)
    else:
        tok = torch.randint(0, 32000, (tokens,), generator=gen, device="cuda")
        tok[: tokens * 7 // 10] = 7
    weight = torch.zeros(32000, cols, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    g = torch.randn(tokens, cols, generator=gen, device="cuda").bfloat16()
    times = {F.embedding: [], fused_ops.embedding: []}
    for rep in range(7):
        for look_up, took in times.items():
            start, end = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            start.record()
            for _ in range(20):
                weight.grad = None
                look_up(tok, weight).backward(g)
            end.record()
            torch.cuda.synchronize()
            took.append(start.elapsed_time(end) / 20)
    theirs, ours = [sorted(t)[3] for t in times.values()]
    assert ours <= theirs, f"{ours * 1e3:.0f} us against {theirs * 1e3:.0f} us"


@pytest.mark.parametrize("ids_dtype", [torch.int64, torch.int32])
def test_embedding_gradient_can_be_differentiated(ids_dtype):
    """A gradient penalty reaches through the table's gradient, as it does through the framework's."""
    gen = torch.Generator(device="cuda").manual_seed(2)
    ids = torch.randint(0, 50, (3, 40), generator=gen, device="cuda").to(ids_dtype)
    w0, g0 = [torch.randn(n, 64, generator=gen, device="cuda").bfloat16() for n in (50, 120)]
    results = []
    for look_up in (fused_ops.embedding, F.embedding):
        w, g = w0.clone().requires_grad_(True), g0.reshape(3, 40, 64).clone().requires_grad_(True)
        (dw,) = torch.autograd.grad(look_up(ids, w), w, g, create_graph=True)
        dw.float().square().sum().backward()
        results.append([dw.detach(), g.grad])
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("tokens,experts,dim", [(1, 8, 64), (333, 64, 256), (8192, 64, 1024), (257, 32, 520)])
def test_router_logits(tokens, experts, dim):
    """The logits are the fp32 GEMM's. Both gradients against 64 bits: one rounding to bf16 (2^-9 of the value, 2^-8 of it allowed) and
    fp32 sums (2^-20 of the sum of the terms' magnitudes), with gradients of the logits over seven orders of magnitude; and no
    further from 64 bits than the library's fp32 GEMMs behind the same rounding."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn(tokens, dim, generator=gen, device="cuda").bfloat16().requires_grad_(True)
    w = (0.05 * torch.randn(experts, dim, generator=gen, device="cuda")).bfloat16().requires_grad_(True)
    g = torch.randn(tokens, experts, generator=gen, device="cuda") * torch.logspace(-6, 1, experts, device="cuda")
    logits = fused_ops.router_logits(x, w)
    logits.backward(g)
    xf, wf = x.detach().float(), w.detach().float()
    assert logits.dtype == torch.float32 and torch.equal(logits.detach(), F.linear(xf, wf))
    xd, wd, gd = xf.double(), wf.double(), g.double()
    for name, got, want, lib, size in (("dx", x.grad, gd @ wd, g @ wf, gd.abs() @ wd.abs()),
                                       ("dw", w.grad, gd.T @ xd, g.T @ xf, gd.abs().T @ xd.abs())):
        err, lib_err = (got.double() - want).abs(), (lib.bfloat16().double() - want).abs()
        assert err.le(2.0**-8 * want.abs() + 2.0**-20 * size).all(), name
        assert torch.linalg.vector_norm(err) <= 1.01 * torch.linalg.vector_norm(lib_err), name


@pytest.mark.parametrize("tokens,experts,dim", [(1, 8, 64), (266, 64, 768), (40, 256, 512), (40, 6, 100)])
def test_router_gradients_are_the_fp32_gemms(tokens, experts, dim):
    """The bits of an fp32 linear layer on widened operands: whatever the number of experts, for infinite and NaN entries (NaN only
    where the sum has one or meets infinities of both signs), and under autocast, which may run it in bf16."""
    gen = torch.Generator(device="cuda").manual_seed(experts)
    x = torch.randn(tokens, dim, generator=gen, device="cuda").bfloat16()
    w = (0.05 * torch.randn(experts, dim, generator=gen, device="cuda")).bfloat16()
    g = torch.randn(tokens, experts, generator=gen, device="cuda")
    for special in (None, 3.4e38, math.inf, math.nan):
        for autocast in (False, True):
            if special is not None:
                g[0, 1], x[-1, 3] = special, special
            grads = []
            for linear in (fused_ops.router_logits, lambda a, b: F.linear(a.float(), b.float())):
                leaves = [t.clone().requires_grad_(True) for t in (x, w)]
                with torch.autocast("cuda", torch.bfloat16, enabled=autocast):
                    out = linear(*leaves)
                out.backward(g.to(out.dtype))
                grads.append([out.detach()] + [t.grad for t in leaves])
            for got, want in zip(*grads):
                assert got.dtype == want.dtype and torch.equal(got.isnan(), want.isnan()), (special, autocast)
                assert torch.equal(got[~got.isnan()], want[~want.isnan()]), (special, autocast)


@pytest.mark.parametrize("layout", ["heads first", "rows first", "odd"])
def test_rope_gradients_of_any_layout(layout):
    """Gradients in the attention's [B, H, S, hd] order, in the projection's [B, S, H, hd] order, and with strides that 16-byte
    accesses cannot take: the same bits."""
    B, S, H, hd = 2, 33, 3, 64
    gen = torch.Generator(device="cuda").manual_seed(1)
    qkv = torch.randn(B, S, 3, H, hd, device="cuda", generator=gen).bfloat16()
    ang = torch.rand(S, hd // 2, device="cuda", generator=gen)
    g = [torch.randn(B, H, S, hd, device="cuda", generator=gen).bfloat16() for _ in range(3)]
    relaid = {"heads first": lambda t: t, "rows first": lambda t: t.transpose(1, 2).contiguous().transpose(1, 2),
              "odd": lambda t: F.pad(t, (1, 2))[..., 1:-2]}[layout]
    grads = []
    for gi in (g, [relaid(t) for t in g]):
        leaf = qkv.clone().requires_grad_(True)
        outs = fused_ops.rope_qkv(leaf, ang.cos(), ang.sin())
        assert all(o.shape == (B, H, S, hd) for o in outs)
        torch.autograd.backward(outs, gi)
        grads.append(leaf.grad)
    assert torch.equal(*grads)


def test_operands_at_any_address():
    """The kernels read 16 bytes at a time; a contiguous view may begin anywhere. Bits of the aligned operands, forward and backward."""
    gen = torch.Generator(device="cuda").manual_seed(31)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()

    def shifted(t):
        view = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)
        assert view.is_contiguous() and view.data_ptr() % 16
        return view

    angles = torch.rand(24, 8, device="cuda", generator=gen)
    targets = torch.randint(0, 264, (33,), device="cuda", generator=gen)
    tokens = torch.randint(0, 50, (70,), device="cuda", generator=gen)
    ops = {
        "norm": (lambda x, w: fused_ops.add_rms_norm(x, None, w, 1e-6), bf(33, 264), bf(264)),
        "add norm": (lambda x, d, w: fused_ops.add_rms_norm(x, d, w, 1e-6), bf(33, 264), bf(33, 264), bf(264)),
        "rope": (lambda qkv, c, s: fused_ops.rope_qkv(qkv, c.detach(), s.detach()), bf(2, 24, 3, 2, 16), angles.cos(), angles.sin()),
        "cross-entropy": (lambda x: fused_ops.cross_entropy(x, targets), bf(33, 264)),
        "swiglu": (lambda x: fused_ops.dense_swiglu(x), bf(33, 528)),
        "embedding": (lambda w: fused_ops.embedding(tokens, w), bf(50, 264)),
        "router": (lambda x, b: fused_ops.router_select(x, b.detach(), 4, 1.5)[1:4:2], bf(33, 64).float(), bf(64).float()),
    }
    for name, (op, *args) in ops.items():
        results, grads = [], None
        for moved in (lambda t: t.clone(), shifted):
            leaves = [moved(t).requires_grad_(True) for t in args]
            out = op(*leaves)
            out = out if isinstance(out, (tuple, list)) else (out,)
            grads = grads or [torch.randn(t.shape, device="cuda", generator=gen).to(t.dtype) for t in out]
            torch.autograd.backward(out, [moved(t) for t in grads])
            results.append([t.detach() for t in out] + [t.grad for t in leaves if t.grad is not None])
        assert len(results[0]) == len(results[1]) > 1, name
        assert all(torch.equal(a, b) for a, b in zip(*results)), name
