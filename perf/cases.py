"""What this framework is timed on: the work its users have it do, at the sizes they do it at.

Everything goes through the public entry points on ONE GPU with every row local (a one-rank expert-parallel group, or
the per-GPU share of a larger one): `chunked_moe` forward and forward + backward, a micro-batch of the decoder trainer,
and the expert kernels on their own. A case is a dict of plain values:

  kind      "train"    forward + backward of the MoE layer; outputs: the layer's output and all four gradients
            "forward"  the layer without autograd (prefill, evaluation, decode); output: the layer's output
            "trainer"  loss and every parameter's gradient of one micro-batch of the DeepSeek-V3-style decoder
            "kernels"  `ops.fused_expert.expert_forward` + `expert_backward` on one expert-major slice
  tokens    tokens of the call (per GPU)          hidden, ffn   model width D and expert width F
  experts   experts on this GPU                   top_k         experts per token
  slice     rows per dispatch slice S             stripe        gate/up stripe width of `w_up`
  wire      "bf16" or "fp8" (`comm_dtype`)        skew          "none", "zipf" or "expert0" (routing imbalance)
  layers    (trainer only) decoder layers, the first one dense. One MoE layer, so that no router reads another MoE
            layer's output: a last-bit difference there can flip a near tie of the top-k and with it whole rows.
"""

import math

import torch

from chunked_ep_moe_b200 import ChunkedMoEConfig, chunked_moe
from chunked_ep_moe_b200.models.deepseek_tiny import DeepSeekTiny, DeepSeekTinyConfig
from chunked_ep_moe_b200.ops import fused_expert

VOCAB = 32000


def _case(name, kind, tokens, hidden, ffn, experts, top_k, slice_rows, stripe=64, wire="bf16", skew="none", layers=0):
    return {"name": name, "kind": kind, "tokens": tokens, "hidden": hidden, "ffn": ffn, "experts": experts,
            "top_k": top_k, "slice": slice_rows, "stripe": stripe, "wire": wire, "skew": skew, "layers": layers}


def listed():
    return [
        # One GPU's share of the DeepSeek-V3-size layer on eight GPUs (32 experts, ~2048 rows each): the largest call.
        _case("train_dsv3_share", "train", 8192, 7168, 2048, 32, 8, 8192),
        # The same layer with few rows per expert (~256), as when one GPU holds many experts of the 256.
        _case("train_dsv3_many_experts", "train", 2048, 7168, 2048, 64, 8, 8192),
        # Rows travel as e4m3 + block scales: the wire option of multi-GPU training.
        _case("train_dsv3_fp8_wire", "train", 4096, 7168, 2048, 32, 8, 8192, wire="fp8"),
        # Imbalanced routing with small slices (the routing stress of the layer): Zipf-distributed expert popularity.
        _case("train_dsv3_zipf", "train", 2999, 7168, 2048, 32, 8, 2048, skew="zipf"),
        # The MoE layer of the small decoder (64 experts of 512, top-6) on one micro-batch of 2 x 4096 tokens.
        _case("train_tiny", "train", 8192, 1024, 512, 64, 6, 16384),
        # A mid-size layer on an odd number of tokens, other stripe width, several small slices.
        _case("train_ragged", "train", 1999, 2048, 1024, 16, 4, 1024, stripe=128),
        # The smallest training call (unit-test sized layers, first steps of a bring-up): launches and host time.
        _case("train_smoke", "train", 192, 256, 256, 8, 2, 128),
        # Prefill / evaluation: forward only, many rows.
        _case("prefill_dsv3", "forward", 4096, 7168, 2048, 32, 8, 8192),
        # Decode with a batch of 64 sequences: ~16 rows per expert, bound by reading the expert weights.
        _case("decode_dsv3_batch", "forward", 64, 7168, 2048, 32, 8, 8192),
        # Decode of a single token on the small decoder's layer: latency.
        _case("decode_tiny_one", "forward", 1, 1024, 512, 64, 6, 8192),
        # Trainer micro-batch: attention, norms, dense and MoE layer, router and loss of the decoder, 2 x 4096 tokens.
        _case("trainer_micro_batch", "trainer", 8192, 1024, 512, 64, 6, 16384, layers=2),
        # The kernel-level surface (what `expert_compute="fused"` runs under a collective transport) on a ragged slice.
        _case("expert_kernels", "kernels", 4001, 2048, 1024, 16, 1, 4096),
    ]


# A drawn layer's weights and GEMM work stay within those of the listed ones.
_MAX_WEIGHTS = 64 * 7168 * 2048
_MAX_WORK = 8192 * 8 * 7168 * 2048


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any kind, sizes spread over their logarithm, odd token counts included."""
    kind = rng.choice(["train"] * 5 + ["forward"] * 3 + ["trainer", "kernels"])
    if kind == "trainer":
        hidden = rng.choice([512, 768, 1024])
        experts = rng.choice([32, 64])
        return {k: v for k, v in _case("", kind, 2 * _log_int(rng, 128, 4096), hidden, rng.choice([256, 512]),
                                       experts, rng.randint(2, 8), rng.choice([4096, 8192, 16384]), layers=2).items()
                if k != "name"}
    while True:
        hidden = 256 * _log_int(rng, 1, 28)
        ffn = 256 * _log_int(rng, 1, 8)
        experts = _log_int(rng, 4, 128)
        top_k = rng.randint(1, min(8, experts))
        tokens = _log_int(rng, 1, 512) if kind == "forward" and rng.random() < 0.6 else _log_int(rng, 64, 8192)
        rows = tokens * top_k
        if experts * hidden * ffn > _MAX_WEIGHTS or rows * hidden * ffn > _MAX_WORK:
            continue
        if kind == "kernels":
            tokens, top_k = min(rows, 16384), 1
            slice_rows = max(8, 8 * math.ceil(tokens * rng.uniform(1.0, 1.3) / 8))
            wire, skew = "bf16", "none"
        else:
            slice_rows = rng.choice([s for s in (512, 1024, 2048, 4096, 8192, 16384) if 24 * s >= rows])
            wire = "fp8" if rng.random() < 0.2 else "bf16"
            skew = rng.choice(["none", "none", "zipf", "expert0"])
        case = _case("", kind, tokens, hidden, ffn, experts, top_k, slice_rows, rng.choice([32, 64, 64, 128]), wire, skew)
        return {k: v for k, v in case.items() if k != "name"}


def _routing(gen, c):
    """Top-k of sigmoid(logits ~ N(0,1)), weights normalised over the chosen ones; `skew` as in routing stress runs."""
    logits = torch.randn(c["tokens"], c["experts"], generator=gen, device="cuda")
    if c["skew"] == "zipf":
        popularity = 1.0 / torch.arange(1, c["experts"] + 1, device="cuda", dtype=torch.float32) ** 1.2
        ids = torch.multinomial(popularity.expand(c["tokens"], c["experts"]), c["top_k"], replacement=False, generator=gen)
        scores = torch.sigmoid(torch.gather(logits, 1, ids))
    else:
        if c["skew"] == "expert0":
            logits[:, 0] += 100.0
        scores, ids = torch.topk(torch.sigmoid(logits), c["top_k"], dim=-1)
    return ids.to(torch.int32), scores / scores.sum(-1, keepdim=True)


def _normal(gen, shape, std=1.0):
    return torch.empty(shape, device="cuda", dtype=torch.bfloat16).normal_(0.0, std, generator=gen)


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    E, D, F, T = c["experts"], c["hidden"], c["ffn"], c["tokens"]
    std = 0.5 / math.sqrt(D)
    if c["kind"] == "trainer":
        cfg = DeepSeekTinyConfig(vocab_size=VOCAB, d_model=D, n_layers=c["layers"], n_heads=D // 64, head_dim=64,
                                 dense_ffn=4 * D, num_experts=E, moe_ffn=F, top_k=c["top_k"], shared_ffn=F,
                                 slice_size=c["slice"], stripe_width=c["stripe"])
        with torch.device("cuda"):
            model = DeepSeekTiny(cfg).to(torch.bfloat16)
        with torch.no_grad():
            for p in model.parameters():
                p.fill_(1.0) if p.dim() == 1 else p.normal_(0.0, cfg.init_std, generator=gen)
        ids = torch.randint(0, VOCAB, (2, T // 2 + 1), generator=gen, device="cuda")
        return {"kind": c["kind"], "model": model, "tokens": ids[:, :-1].contiguous(), "targets": ids[:, 1:].contiguous()}
    w_up, w_down = _normal(gen, (E, D, 2 * F), std), _normal(gen, (E, F, D), std)
    if c["kind"] == "kernels":
        # `tokens` rows dealt to the experts at random, the slice's last rows are padding
        share = torch.multinomial(torch.rand(E, generator=gen, device="cuda") + 0.2, T, replacement=True, generator=gen)
        return {"kind": c["kind"], "groups": torch.bincount(share, minlength=E).to(torch.int32), "rows": T,
                "x": _normal(gen, (c["slice"], D)), "dy": _normal(gen, (c["slice"], D)), "w_up": w_up, "w_down": w_down,
                "stripe": c["stripe"]}
    ids, weights = _routing(gen, c)
    cfg = ChunkedMoEConfig(num_experts=E, top_k=c["top_k"], slice_size=c["slice"], transport="nvshmem",
                           expert_compute="fused", stripe_width=c["stripe"],
                           comm_dtype="float8_e4m3fn" if c["wire"] == "fp8" else None)
    state = {"kind": c["kind"], "cfg": cfg, "x": _normal(gen, (T, D)), "ids": ids, "weights": weights, "w_up": w_up,
             "w_down": w_down}
    if c["kind"] == "train":
        state["g"] = _normal(gen, (T, D))
        for name in ("x", "weights", "w_up", "w_down"):
            state[name].requires_grad_(True)
    return state


def run(s):
    if s["kind"] == "train":
        params = [s["x"], s["weights"], s["w_up"], s["w_down"]]
        for p in params:
            p.grad = None
        out = chunked_moe(s["x"], s["ids"], s["weights"], s["w_up"], s["w_down"], s["cfg"])
        out.backward(s["g"])
        return [out.detach()] + [p.grad for p in params]
    if s["kind"] == "forward":
        with torch.no_grad():
            return chunked_moe(s["x"], s["ids"], s["weights"], s["w_up"], s["w_down"], s["cfg"])
    if s["kind"] == "trainer":
        model = s["model"]
        model.zero_grad(set_to_none=True)
        loss, aux = model(s["tokens"], s["targets"])
        (loss + aux).backward()
        return [loss.detach(), aux.detach()] + [p.grad for p in model.parameters()]
    groups, rows = s["groups"], s["rows"]  # padding rows are not part of any result
    y, res = fused_expert.expert_forward(s["x"], s["w_up"], s["w_down"], groups, stripe=s["stripe"])
    grads = fused_expert.expert_backward(s["x"], s["w_up"], s["w_down"], groups, res, s["dy"], stripe=s["stripe"])
    return [y[:rows], grads.dx[:rows], grads.dw_up, grads.dw_down]


def work(case):
    """Bytes and FLOPs of one pass: inputs once, outputs once, the GEMMs a backward needs without recomputation."""
    c = case
    T, D, F, E, K = c["tokens"], c["hidden"], c["ffn"], c["experts"], c["top_k"]
    if c["kind"] == "trainer":
        dense_params = VOCAB * D + c["layers"] * 4 * D * D + 3 * D * 4 * D + (c["layers"] - 1) * (E * D + 3 * D * F)
        expert_params = (c["layers"] - 1) * 3 * E * D * F
        flops = 6.0 * T * (dense_params + (c["layers"] - 1) * 3 * K * D * F) + c["layers"] * 3 * 1.0 * T * T * D
        return {"bytes": 2.0 * 2 * (dense_params + expert_params + VOCAB * D) + 16.0 * T, "flops": flops}
    rows = T * K
    active = E if c["skew"] != "none" or c["kind"] != "forward" else E * (1.0 - (1.0 - K / E) ** T)
    weights = 3 * D * F * 2.0
    if c["kind"] == "forward":
        return {"bytes": active * weights + 2 * T * D * 2 + rows * 8, "flops": rows * 6.0 * D * F}
    # x, g in; out, dx out; ids, router weights and their gradient; weights in, their gradients out
    return {"bytes": 2 * E * weights + 4 * T * D * 2 + rows * 12, "flops": rows * 18.0 * D * F}


def tolerance(case):
    # bf16 operands and intermediates (h, act, dy, dh) with fp32 accumulation: against an fp32 layer every output of every
    # listed size is off by 0.0022 to 0.0042 (largest difference 0.04 of the value). The trainer adds what its library
    # layers and the embedding's unordered sums do (0.006 against the library's expert layer, 0.002 between two runs).
    return {"rel": 0.02 if case["kind"] == "trainer" else 0.015}
