"""The framework's work as a user's program has it done, one case a size: training steps and inference of a palettized Linear, the
reference's functional API, decoder layers, prefill and decode of whole models, and a served request.

`prepare` makes what a program holds before the call, `run` is one pass through the public entry points, `exact` the same results in
64 bits from plain torch. Sizes are those of the Qwen3-4B decoder layer (width 2560, feed-forward 9728, 32 query and 8 key / value heads of
128), of the hybrid decoders in bench_hybrid.py, and ranges around both.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen-palettize_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import decode_model  # noqa: E402
import decoder_layer  # noqa: E402
import engine  # noqa: E402
import fused_lut_linear_cuda as api  # noqa: E402
import hybrid_model  # noqa: E402
import palettized_linear  # noqa: E402
import plz_ops as ops  # noqa: E402

DEV = "cuda"
GROUP = 256                     # input columns (native layout) or output columns (reference layout) that share a palette
ROOM = 64                       # free positions a decode case keeps behind its cached tokens
VOCAB = 32768
HEAD = 128
# (out features, in features) of the Linears of a decoder layer: gate / up, down, q, o, k / v
SHAPES = ((9728, 2560), (2560, 9728), (4096, 2560), (2560, 4096), (1024, 2560))
# width, feed-forward, query heads, key / value heads, recurrent heads, query latent, key / value latent
MODELS = {"small": (1024, 3072, 16, 8, 8, 512, 256), "medium": (2560, 9728, 32, 8, 20, 1024, 512)}


def listed():
    N, K = SHAPES[0]
    return [
        # the training step of one Linear at the batch of the published configuration (32 x 512 tokens), noise given as a tensor
        {"name": "linear_step_16384", "kind": "linear_step", "M": 16384, "N": N, "K": K, "rank": 16, "noise": "tensor", "straight": True},
        # the same call on a short ragged batch, down projection, larger LoRA rank, sampled noise
        {"name": "linear_step_1000", "kind": "linear_step", "M": 1000, "N": K, "K": N, "rank": 32, "noise": "hash", "straight": True},
        # a program written for the reference: its soft and hard functions under autograd, its tensor layouts
        {"name": "api_soft_2048", "kind": "api_soft", "M": 2048, "N": 4096, "K": 2560, "bias": False},
        {"name": "api_hard_512", "kind": "api_hard", "M": 512, "N": N, "K": K, "bias": True},
        # inference of one Linear for a single token
        {"name": "linear_eval_1", "kind": "linear_eval", "M": 1, "N": N, "K": K, "rank": 0},
        # fine-tuning of a decoder layer with LoRA, forward and backward
        {"name": "layers_8x512", "kind": "layers", "B": 8, "S": 512, "layers": 1, "rank": 16},
        # a batch of prompts through a palettized model
        {"name": "qwen_prefill_4x1024", "kind": "qwen_prefill", "B": 4, "S": 1024, "layers": 2},
        # token decode of a palettized model: one user, and a full batch
        {"name": "qwen_decode_1x2048", "kind": "qwen_decode", "B": 1, "T": 2048, "layers": 4},
        {"name": "qwen_decode_64x1024", "kind": "qwen_decode", "B": 64, "T": 1024, "layers": 4},
        # a hybrid decoder with one layer of each kind: prompts, and a full batch of single tokens
        {"name": "gopunex_prefill_2x1024", "kind": "hybrid_prefill", "design": "Gopunex", "size": "medium", "B": 2, "S": 1024},
        {"name": "gopunex_decode_64x1024", "kind": "hybrid_decode", "design": "Gopunex", "size": "medium", "B": 64, "T": 1024},
        # a request served by the engine: a ragged prompt, then token by token
        {"name": "latodra_request_1000", "kind": "request", "design": "Latodra", "size": "medium", "prompt": 1000, "new": 16},
    ]


def _log(rng, lo, hi):
    """Whole number from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("linear_step", "linear_step", "api_soft", "api_hard", "linear_eval", "linear_eval", "layers", "qwen_prefill", "qwen_decode",
                       "qwen_decode", "hybrid_prefill", "hybrid_decode", "hybrid_decode", "request"))
    N, K = rng.choice(SHAPES)
    c = {"kind": kind}
    if kind == "linear_step":
        c.update(M=_log(rng, 64, 8192), N=N, K=K, rank=rng.choice((16, 32)), noise=rng.choice(("tensor", "hash")), straight=rng.random() < 0.75)
    elif kind == "api_soft":
        c.update(M=_log(rng, 16, 4096), N=N, K=K, bias=rng.random() < 0.5)
    elif kind == "api_hard":
        c.update(M=_log(rng, 16, 8192), N=N, K=K, bias=rng.random() < 0.5)
    elif kind == "linear_eval":
        c.update(M=_log(rng, 1, 4096), N=N, K=K, rank=rng.choice((0, 0, 16)))
    elif kind == "layers":
        c.update(B=_log(rng, 1, 8), S=128 * rng.randint(1, 4), layers=1, rank=rng.choice((16, 32)))
    elif kind == "qwen_prefill":
        c.update(B=_log(rng, 1, 4), S=128 * rng.randint(1, 8), layers=rng.randint(1, 2))
    elif kind == "qwen_decode":
        c.update(B=_log(rng, 1, 64), T=_log(rng, 16, 2048), layers=rng.randint(1, 4))
    else:
        c.update(design=rng.choice(("Gopunex", "Latodra")), size=rng.choice(("small", "medium")))
        if kind == "hybrid_prefill":
            c.update(B=_log(rng, 1, 2), S=_log(rng, 65, 1024))
        elif kind == "hybrid_decode":
            c.update(B=_log(rng, 1, 64), T=_log(rng, 16, 2048))
        else:
            c.update(prompt=_log(rng, 16, 1024), new=rng.randint(4, 24))
    return c


# ---- inputs, from the seed alone ---------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(torch.bfloat16)


def _palette(g, groups):
    """Sorted 4-tuples of N(0, 0.02^2)."""
    return (torch.randn(groups, 4, generator=g, device=DEV) * 0.02).sort(-1).values.to(torch.bfloat16)


def _gumbel(g, *shape):
    u = torch.rand(*shape, generator=g, device=DEV).clamp_(min=1e-7, max=1.0 - 2.0 ** -24)
    return u.log_().neg_().log_().neg_()


def _linear_inputs(c, seed):
    g, M, N, K = _gen(seed), c["M"], c["N"], c["K"]
    d = {"x": _randn(g, M, K)}
    if c["kind"] == "linear_step":
        d.update(dy=_randn(g, M, N), palette=_palette(g, N * (K // GROUP)), logits=torch.randn(N, K, 4, generator=g, device=DEV))
        d["noise"] = _gumbel(g, N, K, 4) if c["noise"] == "tensor" else "hash"
    elif c["kind"] == "linear_eval":
        d.update(palette=_palette(g, N * (K // GROUP)), logits=torch.randn(N, K, 4, generator=g, device=DEV))
    else:
        d.update(dy=_randn(g, M, N), palette=_palette(g, N // GROUP), bias=_randn(g, N, scale=0.1) if c["bias"] else None)
        if c["kind"] == "api_soft":
            d.update(logits=torch.randn(4, K, N, generator=g, device=DEV).half(), noise=_gumbel(g, 4, K, N))
        else:
            d["indices"] = torch.randint(0, 4, (K, N), generator=g, device=DEV, dtype=torch.int8)
    if c.get("rank"):
        d.update(A=_randn(g, c["rank"], K, scale=K ** -0.5), B=_randn(g, N, c["rank"], scale=0.01))
    return d


def _layer_inputs(cfg, seed, layers, rank=0):
    """Indices, palettes, LoRA factors and norm weights of every layer, by name."""
    g, out = _gen(seed), []
    for _ in range(layers):
        L = {}
        for name, (N, K) in cfg.shapes().items():
            L[name] = {"idx": torch.randint(0, 4, (N, K), generator=g, device=DEV, dtype=torch.int8), "palette": _palette(g, N * (K // GROUP))}
            if rank:
                L[name].update(A=_randn(g, rank, K, scale=K ** -0.5), B=_randn(g, N, rank, scale=0.01))
        for name, n in (("input_ln", cfg.hidden), ("post_ln", cfg.hidden), ("q_norm", HEAD), ("k_norm", HEAD)):
            L[name] = (1.0 + 0.1 * torch.randn(n, generator=g, device=DEV)).to(torch.bfloat16)
        out.append(L)
    return g, out


def _packed(e, cfg, name):
    N, K = cfg.shapes()[name]
    return ops.PackedWeight(ops.pack_indices(e["idx"], n_major=True), e["palette"], N, K, 1, GROUP)


def _qwen_inputs(c, seed):
    cfg = decode_model.ModelConfig(n_layers=c["layers"], vocab=VOCAB)
    g, L = _layer_inputs(cfg, seed, c["layers"])
    d = {"cfg": cfg, "layers": L, "embed": _randn(g, VOCAB, cfg.hidden, scale=0.02), "norm": (1.0 + 0.1 * torch.randn(cfg.hidden, generator=g, device=DEV)).to(torch.bfloat16)}
    if c["kind"] == "qwen_prefill":
        d["ids"] = torch.randint(0, VOCAB, (c["B"], c["S"]), generator=g, device=DEV)
    else:
        shape = (c["layers"], c["B"], c["T"] + ROOM, cfg.n_kv_heads * HEAD)
        d.update(ids=torch.randint(0, VOCAB, (c["B"], 1), generator=g, device=DEV), k=_randn(g, *shape), v=_randn(g, *shape))
    return d


def _hybrid_config(c):
    width, ff, H, G, R, rq, rkv = MODELS[c["size"]]
    if c["design"] == "Gopunex":
        mix = [("lightning", {"decay": [0.9 + 0.099 * i / R for i in range(R)], "dim": HEAD, "heads": R, "vdim": HEAD}),
               ("channel_delta", {"conv": 4, "dim": HEAD, "heads": R, "kv_heads": R, "vdim": HEAD}),
               ("attention", {"bias_max": 512, "dim": HEAD, "heads": H, "kv_heads": G, "scale": HEAD ** -0.5, "v_mix": True, "vdim": HEAD})]
        out = {"embedding": {"scale": 1.0}, "residual_mult": 0.7}
    else:
        plain = {"dim": HEAD, "heads": H, "kv_rank": rkv, "q_rank": rq, "vdim": HEAD}
        rot = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "fast": 32.0, "original": 4096, "slow": 1.0}}
        mix, out = [("latent_attention", {**plain, "rot_dim": 64, "scale": 192 ** -0.5, "rot": rot}), ("latent_attention_2", {**plain, "scale": HEAD ** -0.5})], {}
    out.update(architecture=c["design"], norm={"eps": 1e-6}, vocab=VOCAB, width=width,
               layers=[{"type": t, "mixer": m, "mlp": {"ff": ff, "kind": "dense"}} for t, m in mix])
    return out


def _hybrid_state(cfg, B, T, g):
    """What the layers keep for sequences of T tokens, with room for ROOM more: a dict of tensors for each layer."""
    out = []
    for e in cfg["layers"]:
        m = e["mixer"]
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        if e["type"] == "attention":
            st = {"k": _randn(g, B, T + ROOM, m["kv_heads"] * dk), "v": _randn(g, B, T + ROOM, m["kv_heads"] * dv)}
        elif "kv_rank" in m:
            st = {"c": _randn(g, B, T + ROOM, m["kv_rank"])}
            if "rot_dim" in m:
                st["kr"] = _randn(g, B, T + ROOM, m["rot_dim"])
        else:
            st = {"S": torch.randn(B, H, dk, dv, generator=g, device=DEV)}
            if "conv" in m:
                st["conv"] = _randn(g, B, m["conv"] - 1, 2 * m["kv_heads"] * dk + H * dv)
        out.append(st)
    return out


def _hybrid_inputs(c, seed):
    cfg, g = _hybrid_config(c), _gen(seed)
    d = {"cfg": cfg, "weights": hybrid_model.random_tensors(cfg, seed, DEV)}
    if c["kind"] == "hybrid_prefill":
        d["ids"] = torch.randint(0, VOCAB, (c["B"], c["S"]), generator=g, device=DEV)
    elif c["kind"] == "hybrid_decode":
        d.update(ids=torch.randint(0, VOCAB, (c["B"], 1), generator=g, device=DEV), state=_hybrid_state(cfg, c["B"], c["T"], g))
    else:
        d["ids"] = torch.randint(0, VOCAB, (1, c["prompt"] + c["new"]), generator=g, device=DEV)
    return d


# ---- the calls -----------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind in ("linear_step", "linear_eval", "api_soft", "api_hard"):
        d = _linear_inputs(c, seed)
        if kind == "linear_eval":
            m = palettized_linear.PalettizedLinear(c["K"], c["N"], rank=c["rank"], lora_scale=2.0, device=DEV)
            with torch.no_grad():
                m.index_logits.copy_(d["logits"])
                m.palette.copy_(d["palette"].view(m.palette.shape))
                if c["rank"]:
                    m.lora_A.copy_(d["A"])
                    m.lora_B.copy_(d["B"])
            m.extract_hard_indices()
            s.update(x=d["x"], module=m.eval())
        else:
            if kind != "linear_step":
                for name in ("x", "palette", "logits", "bias"):
                    if d.get(name) is not None:
                        d[name].requires_grad_(True)
            elif c["rank"]:
                d["lora"] = (d["A"], d["B"], 2.0)
            s.update(d)
    elif kind == "layers":
        cfg = decoder_layer.LayerConfig(lora_rank=c["rank"])
        g, L = _layer_inputs(cfg, seed, c["layers"], c["rank"])
        s["layers"] = [decoder_layer.LayerParams({n: decoder_layer.PalettizedLoraLinear(_packed(e[n], cfg, n), e[n]["A"], e[n]["B"], cfg.lora_scale) for n in decoder_layer.LINEARS},
                                                 e["input_ln"], e["post_ln"], e["q_norm"], e["k_norm"]) for e in L]
        s.update(cfg=cfg, x=_randn(g, c["B"] * c["S"], cfg.hidden), dy=_randn(g, c["B"] * c["S"], cfg.hidden))
        s["cos"], s["sin"] = ops.rope_tables(c["S"], HEAD, cfg.rope_theta, DEV)
    elif kind in ("qwen_prefill", "qwen_decode"):
        d = _qwen_inputs(c, seed)
        cfg = d["cfg"]
        L = [{n: _packed(e[n], cfg, n) if n in decoder_layer.LINEARS else e[n] for n in e} for e in d["layers"]]
        s["model"] = decode_model.PalettizedQwen(cfg, L, d["embed"], d["norm"], max_positions=4096)
        s["ids"] = d["ids"]
        if kind == "qwen_prefill":
            s["cache"] = s["model"].new_cache(c["B"], c["S"])
        else:
            s["cache"] = decode_model.KVCache(d["k"], d["v"], c["T"])
    else:
        d = _hybrid_inputs(c, seed)
        model = hybrid_model.ARCHITECTURES[c["design"]].from_config(d["cfg"], d["weights"], torch.bfloat16, DEV)
        s["model"] = model
        if kind == "request":
            s["engine"] = engine.Engine(model, max_tokens=c["prompt"] + c["new"])
            s["tokens"] = d["ids"][0].tolist()
        else:
            s["ids"] = d["ids"]
            s["cache"] = model.new_cache(c["B"], c["S"] if kind == "hybrid_prefill" else c["T"] + ROOM)
            if kind == "hybrid_decode":
                for kept, given in zip(s["cache"].layers, d["state"]):
                    for name, t in given.items():
                        kept[name].copy_(t)
                s["cache"].length = c["T"]
                s["cache"].pos.fill_(c["T"])
    return s


def _written(cache, first, n):
    """What a step over the positions first .. first + n - 1 leaves in a hybrid decoder's state."""
    return [{name: t if name in ("S", "conv") else t[:, first:first + n] for name, t in st.items()} for st in cache.layers]


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "linear_step":
        return palettized_linear.linear_step(s["x"], s["dy"], s["palette"], s["logits"], s["noise"], 1.0, lora=s.get("lora"), ste=c["straight"], seed=7)
    if kind == "linear_eval":
        return s["module"](s["x"]).detach()
    if kind == "api_soft":
        y = api.fused_lut_linear_soft(s["x"], s["palette"], s["logits"], s["bias"], GROUP, 1.0, noise=s["noise"])
        want = [t for t in (s["x"], s["palette"], s["logits"], s["bias"]) if t is not None]
        return [y.detach(), *torch.autograd.grad(y, want, s["dy"])]
    if kind == "api_hard":
        y = api.fused_lut_linear(s["x"], s["palette"], s["indices"], s["bias"], GROUP)
        want = [t for t in (s["x"], s["palette"], s["bias"]) if t is not None]
        return [y.detach(), *torch.autograd.grad(y, want, s["dy"])]
    if kind == "layers":
        y, dx, grads = decoder_layer.stack_forward_backward(s["cfg"], s["layers"], s["x"], s["dy"], c["B"], c["S"], s["cos"], s["sin"])
        return {"y": y, "dx": dx, "grads": grads}
    cache = s.get("cache")
    if kind == "qwen_prefill":
        cache.reset()
        h, logits = s["model"].prefill(s["ids"], cache)
        return {"h": h, "logits": logits, "k": cache.k, "v": cache.v}
    if kind == "hybrid_prefill":
        cache.reset()
        logits = s["model"].prefill(s["ids"], cache)
        return {"logits": logits, "state": _written(cache, 0, c["S"])}
    if kind == "request":
        at, tokens, out = c["prompt"], s["tokens"], []
        out.append(s["engine"].step("r", tokens[:at], [at - 1]))
        for t in range(at, len(tokens)):
            out.append(s["engine"].step("r", [tokens[t]], [0], end=t + 1 == len(tokens)))
        return {"logits": torch.cat(out)}
    if cache.length == cache.capacity:          # the room is used up: back to the cached tokens
        cache.length = c["T"]
        if kind == "hybrid_decode":
            cache.pos.fill_(c["T"])
    first = cache.length
    if kind == "qwen_decode":
        logits = s["model"].decode_step(s["ids"][:, 0], cache)
        return {"logits": logits, "k": cache.k[:, :, first], "v": cache.v[:, :, first]}
    logits = s["model"].decode_step(s["ids"][:, 0], cache)
    return {"logits": logits, "state": _written(cache, first, 1)}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def _hybrid_weights(cfg):
    """Elements of all matrices (embedding aside, head included)."""
    return sum(math.prod(s) for n, s in hybrid_model.tensor_shapes(cfg).items() if len(s) == 2 and n != "embed") + (cfg["vocab"] * cfg["width"] if cfg["architecture"] == "Latodra" else 0)


def _mixing(e, past, n):
    """(FLOPs, bytes per sequence and position read) of what lies between a layer's projections, for n tokens behind `past` of one sequence."""
    m, pairs = e["mixer"], n * past + n * (n + 1) / 2
    H, dk, dv = m["heads"], m["dim"], m["vdim"]
    if e["type"] == "attention":
        return 2 * pairs * H * (dk + dv), 2 * m["kv_heads"] * (dk + dv) * (past + n), 0
    if "kv_rank" in m:
        per = m["kv_rank"] + m.get("rot_dim", 0)
        return 2 * pairs * H * (dk + m.get("rot_dim", 0) + dv), 2 * per * (past + n), 0
    return 6 * n * H * dk * dv, 0, 4 * H * dk * dv * (2 if past else 1)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("linear_step", "linear_eval", "api_soft", "api_hard"):
        M, N, K, r = c["M"], c["N"], c["K"], c.get("rank", 0)
        gemm, lora, io, pal = 2 * M * N * K, 2 * M * r * (N + K), 2 * M * (N + K), 8 * N * K // GROUP
        if kind == "linear_eval":
            return {"bytes": N * K / 4 + pal + io + 2 * r * (N + K), "flops": gemm + lora}
        if kind == "api_hard":
            return {"bytes": N * K / 4 + 2 * io, "flops": 3 * gemm}
        per = 16 + 16 + (0 if c.get("noise") == "hash" else 16) if kind == "linear_step" else 8 + 8 + 16
        return {"bytes": per * N * K + 2 * io + (2 * pal if kind == "linear_step" else 0) + 6 * r * (N + K), "flops": 3 * gemm + 3 * lora}
    if kind in ("layers", "qwen_prefill", "qwen_decode"):
        cfg = decode_model.ModelConfig()
        n_w, L, B = sum(N * K for N, K in cfg.shapes().values()), c["layers"], c["B"]
        kv = 4 * cfg.n_kv_heads * HEAD
        if kind == "layers":
            M, r = B * c["S"], c["rank"]
            lora = r * sum(N + K for N, K in cfg.shapes().values())
            att = 2 * B * c["S"] ** 2 * cfg.n_heads * HEAD
            return {"bytes": L * (n_w / 4 + n_w / 32 + n_w / 16 + 6 * lora) + 8 * M * cfg.hidden, "flops": L * (6 * M * (n_w + lora) + 3.5 * att)}
        if kind == "qwen_prefill":
            M, att = B * c["S"], 2 * B * c["S"] ** 2 * cfg.n_heads * HEAD
            return {"bytes": L * (n_w / 4 + n_w / 32 + M * kv) + 2 * VOCAB * cfg.hidden + 4 * M * cfg.hidden, "flops": L * (2 * M * n_w + att) + 2 * B * VOCAB * cfg.hidden}
        return {"bytes": L * (n_w / 4 + n_w / 32 + B * c["T"] * kv) + 2 * VOCAB * cfg.hidden + 2 * B * VOCAB,
                "flops": 2 * B * (L * n_w + VOCAB * cfg.hidden) + L * 4 * B * c["T"] * cfg.n_heads * HEAD}
    cfg = _hybrid_config(c)
    n_w, head = _hybrid_weights(cfg), cfg["vocab"] * cfg["width"]
    B, steps = c.get("B", 1), [(0, c["S"])] if kind == "hybrid_prefill" else [(c["T"], 1)] if kind == "hybrid_decode" else [(0, c["prompt"])] + [(c["prompt"] + i, 1) for i in range(c["new"])]
    out = {"bytes": 0.0, "flops": 0.0}
    for past, n in steps:
        out["bytes"] += 2 * n_w + B * (4 * n * cfg["width"] + 4 * cfg["vocab"])
        out["flops"] += 2 * B * (n * (n_w - head) + head)
        for e in cfg["layers"]:
            fl, cached, kept = _mixing(e, past, n)
            out["flops"] += B * fl
            out["bytes"] += B * (cached + kept)
    return out


def tolerance(case):
    """Four times the distance from the same in 64 bits: 0.0017 where one bf16 rounding lies between input and output, 0.006 for a layer forward
    and backward, 0.017 for the logits of palettized layers in a row (0.03 is the most that is allowed), 0.005 for the hybrid decoders, whose
    residual stream is fp32."""
    kind = case["kind"]
    if kind in ("linear_step", "linear_eval", "api_soft", "api_hard"):
        return {"rel": 0.007}
    if kind == "layers":
        return {"rel": 0.025}
    return {"rel": 0.03 if kind in ("qwen_prefill", "qwen_decode") else 0.02}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("linear_step", "linear_eval", "api_soft", "api_hard"):
        return _exact_linear(case, _linear_inputs(case, seed))
    if kind == "layers":
        return _exact_layers(case, seed)
    if kind in ("qwen_prefill", "qwen_decode"):
        return _exact_qwen(case, _qwen_inputs(case, seed))
    d = _hybrid_inputs(case, seed)
    if kind == "hybrid_prefill":
        h, state = _hybrid_forward(d["cfg"], d["weights"], d["ids"], None, 0)
        return {"logits": _hybrid_logits(d["cfg"], d["weights"], h[:, -1]), "state": state}
    if kind == "hybrid_decode":
        h, state = _hybrid_forward(d["cfg"], d["weights"], d["ids"], d["state"], case["T"])
        return {"logits": _hybrid_logits(d["cfg"], d["weights"], h[:, -1]), "state": state}
    h, _ = _hybrid_forward(d["cfg"], d["weights"], d["ids"], None, 0)
    return {"logits": _hybrid_logits(d["cfg"], d["weights"], h[0, case["prompt"] - 1:])}


def _hash_noise(seed, N, K):
    """The counter-based Gumbel sampler: a 32-bit hash of ((k * N + n) * 4 + entry), its low 24 bits as a uniform number."""
    k, n, e = (torch.arange(m, dtype=torch.int64, device=DEV) for m in (K, N, 4))
    i = ((k[None, :, None] * N + n[:, None, None]) * 4 + e) & 0xFFFFFFFF
    m32 = 0xFFFFFFFF
    i = seed ^ (i * 0x9E3779B9 & m32)
    i ^= i >> 13
    i = (i * 1103515245 + 12345) & m32
    i ^= i >> 17
    i = (i * 1103515245 + 12345) & m32
    u = ((i & 0xFFFFFF).double() / 16777216.0).clamp_(min=float(np.float32(1e-7)))
    return u.log_().neg_().log_().neg_()


def _spread(palette, N, K, gs_n, gs_k):
    """Palette entries [N, K / gs_k, 4] of every output row and column group."""
    return palette.detach().double().view(N // gs_n, K // gs_k, 4).repeat_interleave(gs_n, 0)


def _pick(pal, idx, gs_k):
    """W [N, K] from the entries of _spread and the indices."""
    N, K = idx.shape
    return torch.gather(pal[:, :, None, :].expand(-1, -1, gs_k, -1).reshape(N, K, 4), 2, idx.long()[:, :, None])[:, :, 0]


def _exact_linear(c, d):
    M, N, K, kind = c["M"], c["N"], c["K"], c["kind"]
    native = kind in ("linear_step", "linear_eval")
    gs_n, gs_k = (1, GROUP) if native else (GROUP, K)
    x, pal = d["x"].double(), _spread(d["palette"], N, K, gs_n, gs_k)
    logits = d["logits"] if native else d["logits"].permute(2, 1, 0) if kind == "api_soft" else None
    idx = d["indices"].T if logits is None else logits.argmax(-1)
    P = None
    if kind in ("linear_step", "api_soft"):
        noise = _hash_noise(7, N, K) if d["noise"] is None or isinstance(d["noise"], str) else d["noise"] if native else d["noise"].permute(2, 1, 0)
        P = torch.softmax(logits.double() + noise.double(), -1)
        del noise
        soft = torch.einsum("nkjp,nkp->nkj", P.view(N, K // gs_k, gs_k, 4), pal).reshape(N, K)
    W = _pick(pal, idx, gs_k) if c.get("straight", True) else soft
    y = x @ W.T
    if c.get("rank"):
        A, B = d["A"].double(), d["B"].double()
        t = 2.0 * x @ A.T
        y += t @ B.T
    if d.get("bias") is not None:
        y += d["bias"].detach().double()
    if kind == "linear_eval":
        return y
    dy = d["dy"].double()
    dx, dW = dy @ W, dy.T @ x
    if kind == "api_hard":
        hot = torch.nn.functional.one_hot(idx.long(), 4).double()
        out = [y, dx, torch.einsum("nk,nkp->np", dW, hot).view(N // GROUP, GROUP, 4).sum(1)]
        return out + [dy.sum(0)] if d["bias"] is not None else out
    dpal = torch.einsum("nkj,nkjp->nkp", dW.view(N, K // gs_k, gs_k), P.view(N, K // gs_k, gs_k, 4))
    dlog = P
    for i in range(0, N, 512):                                 # in place, in row blocks: the entries are large
        e = pal[i:i + 512, :, None, :].expand(-1, -1, gs_k, -1).reshape(-1, K, 4)
        dlog[i:i + 512] *= (e - soft[i:i + 512, :, None]) * dW[i:i + 512, :, None]
    if native:
        dt = 2.0 * dy @ B
        return {"packed": None, "y": y, "dx": dx + dt @ A, "dlogits": dlog, "dpalette": dpal.view(-1, 4), "da": dt.T @ x, "db": dy.T @ t}
    out = [y, dx, dpal.view(N // GROUP, GROUP, 4).sum(1), dlog.permute(2, 1, 0)]
    return out + [dy.sum(0)] if d["bias"] is not None else out


def _rms(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v, scale, bias=None, sink=None):
    """Causal attention of the last q.shape[1] positions: q [B, n, H, d], k, v [B, T, G, .]; bias [H, distances]; sink [H] scores."""
    B, n, H, _ = q.shape
    T, G = k.shape[1], k.shape[2]
    at = torch.arange(T - n, T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None, :]
    out = []
    for b in range(B):
        s = torch.einsum("ngrd,tgd->grnt", q[b].reshape(n, G, H // G, -1), k[b]).reshape(H, n, T) * scale
        if bias is not None:
            s = s + bias[:, at.clamp(0, bias.shape[1] - 1)]
        s = s.masked_fill(at < 0, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, n, 1)], -1)
        p = torch.softmax(s, -1)[:, :, :T]
        out.append(torch.einsum("grnt,tgd->ngrd", p.view(G, H // G, n, T), v[b]).reshape(n, -1))
    return torch.stack(out)


def _rope(x, first):
    """Rotate-half positions first .. of x [B, n, heads, 128], the angles as the 32-bit tables hold them."""
    f = 1.0 / (1e6 ** (torch.arange(0, HEAD, 2).float() / HEAD))
    a = (torch.arange(first, first + x.shape[1]).float()[:, None] * f).to(DEV)
    cos, sin = (torch.cat([t, t], -1).double()[:, None] for t in (a.cos(), a.sin()))
    return x * cos + torch.cat([-x[..., HEAD // 2:], x[..., :HEAD // 2]], -1) * sin


def _qwen_layer(cfg, W, lin, x, past_k, past_v, first):
    """One decoder layer in 64 bits: x [B, n, hidden] -> (x, new keys, new values)."""
    B, n, _ = x.shape
    h = _rms(x, W["input_ln"])
    q = _rope(_rms(lin("q", h).view(B, n, cfg.n_heads, HEAD), W["q_norm"]), first)
    k = _rope(_rms(lin("k", h).view(B, n, cfg.n_kv_heads, HEAD), W["k_norm"]), first)
    v = lin("v", h).view(B, n, cfg.n_kv_heads, HEAD)
    kk, vv = (k, v) if past_k is None else (torch.cat([p.double().view(B, -1, cfg.n_kv_heads, HEAD), t], 1) for p, t in ((past_k, k), (past_v, v)))
    x = x + lin("o", _attend(q, kk, vv, HEAD ** -0.5))
    h = _rms(x, W["post_ln"])
    return x + lin("down", torch.nn.functional.silu(lin("gate", h)) * lin("up", h)), k.reshape(B, n, -1), v.reshape(B, n, -1)


def _dense(e):
    N, K = e["idx"].shape
    return _pick(_spread(e["palette"], N, K, 1, GROUP), e["idx"], GROUP)


def _exact_qwen(c, d):
    cfg, B = d["cfg"], c["B"]
    x, ks, vs = d["embed"].double()[d["ids"]], [], []
    first = c.get("T", 0)
    for i, L in enumerate(d["layers"]):
        W = {n: t.double() for n, t in L.items() if isinstance(t, torch.Tensor)}
        past = (d["k"][i, :, :first], d["v"][i, :, :first]) if first else (None, None)
        x, k, v = _qwen_layer(cfg, W, lambda n, h: h @ _dense(L[n]).T, x, *past, first)
        ks.append(k)
        vs.append(v)
    logits = _rms(x[:, -1], d["norm"].double()) @ d["embed"].double().T
    k, v = torch.stack(ks), torch.stack(vs)
    if c["kind"] == "qwen_decode":
        return {"logits": logits, "k": k[:, :, 0], "v": v[:, :, 0]}
    return {"h": x.view(B * c["S"], -1), "logits": logits, "k": k, "v": v}


def _exact_layers(c, seed):
    cfg = decoder_layer.LayerConfig(lora_rank=c["rank"])
    g, layers = _layer_inputs(cfg, seed, c["layers"], c["rank"])
    x, dy = (_randn(g, c["B"] * c["S"], cfg.hidden).double().view(c["B"], c["S"], -1) for _ in range(2))
    leaves, h = [], x.requires_grad_(True)
    for L in layers:
        W = {n: t.double().requires_grad_(True) for n, t in L.items() if isinstance(t, torch.Tensor)}
        for n in decoder_layer.LINEARS:
            W[n] = {k: L[n][k].double().requires_grad_(True) for k in ("palette", "A", "B")}
        leaves.append(W)

        def lin(n, z, W=W, L=L):
            N, K = L[n]["idx"].shape
            w = torch.gather(W[n]["palette"].view(N, K // GROUP, 4), 2, L[n]["idx"].long().view(N, K // GROUP, GROUP)).view(N, K)
            return z @ w.T + cfg.lora_scale * (z @ W[n]["A"].T) @ W[n]["B"].T
        h, _, _ = _qwen_layer(cfg, W, lin, h, None, None, 0)
    h.backward(dy)
    grads = [{n: tuple(t.grad for t in w.values()) if isinstance(w, dict) else w.grad for n, w in W.items()} for W in leaves]
    return {"y": h.detach().view(-1, cfg.hidden), "dx": x.grad.view(-1, cfg.hidden), "grads": grads}


def _silu(x):
    return torch.nn.functional.silu(x)


def _lightning(h, W, m, st):
    B, n, _ = h.shape
    H, dk, dv = m["heads"], m["dim"], m["vdim"]
    q, k, v = (_silu(h @ W(t).T).view(B, n, H, -1) for t in "qkv")
    S = torch.zeros(B, H, dk, dv, dtype=torch.float64, device=DEV) if st is None else st["S"].double()
    decay, o = torch.tensor(m["decay"], dtype=torch.float32, device=DEV).double()[None, :, None, None], []
    for t in range(n):
        S = decay * S + k[:, t, :, :, None] * v[:, t, :, None, :]
        o.append(torch.einsum("bhk,bhkv->bhv", q[:, t], S))
    o = _rms(torch.stack(o, 1).view(B, n, H * dv), W("norm"))
    return (o * torch.sigmoid(h @ W("g").T)) @ W("o").T, {"S": S}


def _channel_delta(h, W, m, st):
    B, n, _ = h.shape
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    raw = torch.cat([h @ W(t).T for t in "qkv"], -1)
    before = torch.zeros(B, taps - 1, raw.shape[2], dtype=torch.float64, device=DEV) if st is None else st["conv"].double()
    raw = torch.cat([before, raw], 1)
    w = torch.cat([W(t + ".conv") for t in "qkv"])
    q, k, v = _silu(sum(raw[:, i:i + n] * w[:, i] for i in range(taps))).split([G * dk, G * dk, H * dv], -1)

    def unit(z):
        z = z.view(B, n, G, dk)
        return (z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)
    q, k, v = unit(q) * dk ** -0.5, unit(k), v.view(B, n, H, dv)
    beta = torch.sigmoid(h @ W("b").T)
    g = torch.nn.functional.softplus((h @ W("a1").T) @ W("a2").T + W("dt_bias")).view(B, n, H, dk)
    g = torch.exp(-torch.exp(W("A_log"))[:, None] * g)
    S = torch.zeros(B, H, dk, dv, dtype=torch.float64, device=DEV) if st is None else st["S"].double()
    o = []
    for t in range(n):
        S = g[:, t, :, :, None] * S
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhk,bhkv->bhv", k[:, t], S))
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        o.append(torch.einsum("bhk,bhkv->bhv", q[:, t], S))
    gate = torch.sigmoid((h @ W("g1").T) @ W("g2").T).view(B, n, H, dv)
    return (_rms(torch.stack(o, 1), W("norm")) * gate).reshape(B, n, -1) @ W("o").T, {"S": S, "conv": raw[:, n:]}


def _bias_attention(h, W, m, st, first):
    B, n, _ = h.shape
    H, G, dk, dv, rel = m["heads"], m["kv_heads"], m["dim"], m["vdim"], W("rel")
    q, k, v = (h @ W(t).T + W(t + ".b") for t in "qkv")
    q, k = _rms(q, W("q.norm")), _rms(k, W("k.norm"))
    half, far = rel.shape[0] // 2, m["bias_max"]
    row = [d if d < half else min(2 * half - 1, half + math.floor(math.log(d / half) / math.log(far / half) * half + 1e-9)) for d in range(far + 1)]
    kk, vv = (k, v) if st is None else (torch.cat([st[t][:, :first].double(), z], 1) for t, z in (("k", k), ("v", v)))
    o = _attend(q.view(B, n, H, dk), kk.view(B, -1, G, dk), vv.view(B, -1, G, dv), m["scale"], rel[row].T, torch.zeros(H, dtype=torch.float64, device=DEV))
    return o @ W("o").T, {"k": k, "v": v}


def _turn(x, first, rot):
    """x [B, n, ..., dims]: pairs (2 i, 2 i + 1) turned by position * frequency i (YaRN)."""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    place = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEV)
    slow = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f = base ** (-2.0 * i / dims) * (slow / sc["factor"] + 1.0 - slow)
    a = torch.arange(first, first + x.shape[1], dtype=torch.float64, device=DEV)[:, None] * f
    size = 0.1 * math.log(sc["factor"]) + 1.0
    cos, sin = (t.view(1, x.shape[1], *[1] * (x.dim() - 3), dims // 2) * size for t in (a.cos(), a.sin()))
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)


def _latent_attention(h, W, m, st, first):
    B, n, _ = h.shape
    H, dn, dv, R, dr = m["heads"], m["dim"], m["vdim"], m["kv_rank"], m.get("rot_dim", 0)
    q = (_rms(h @ W("dq").T, W("dq.norm")) @ W("uq").T).view(B, n, H, dn + dr)
    low = h @ W("dkv").T
    new = {"c": _rms(low[..., :R], W("dkv.norm"))}
    if dr:
        new["kr"] = _turn(low[..., R:], first, m["rot"])
        q = torch.cat([q[..., :dn], _turn(q[..., dn:], first, m["rot"])], -1)
    have = new if st is None else {t: torch.cat([st[t][:, :first].double(), new[t]], 1) for t in new}
    o = []
    for b in range(B):                                         # keys and values of every head of one sequence at a time
        k, v = ((have["c"][b] @ W(t).T).view(1, -1, H, d) for t, d in (("uk", dn), ("uv", dv)))
        if dr:
            k = torch.cat([k, have["kr"][b][None, :, None].expand(-1, -1, H, -1)], -1)
        o.append(_attend(q[b:b + 1], k, v, m["scale"], None, W("sink") if dr else None))
    o = torch.cat(o)
    return (o if dr else o * torch.sigmoid(h @ W("g").T)) @ W("o").T, new


def _hybrid_forward(cfg, weights, ids, state, first):
    """Residual stream [B, n, width] after all layers, and what the step leaves in the state."""
    latodra, kept = cfg["architecture"] == "Latodra", []
    top = lambda name: weights[name].double()
    x = top("embed")[ids]
    if latodra:
        x = _rms(x, top("embed.norm"))
    for i, e in enumerate(cfg["layers"]):
        W, st, p = lambda name, i=i: weights[f"l{i}.mix.{name}"].double(), None if state is None else state[i], f"l{i}."
        mix = {"lightning": lambda h: _lightning(h, W, e["mixer"], st), "channel_delta": lambda h: _channel_delta(h, W, e["mixer"], st),
               "attention": lambda h: _bias_attention(h, W, e["mixer"], st, first)}.get(e["type"], lambda h: _latent_attention(h, W, e["mixer"], st, first))
        if latodra:
            y, new = mix(_rms(x, top(p + "norm1")))
            x = x + _rms(y, top(p + "norm1b")) * top(p + "ls1")
            h = _rms(x, top(p + "norm2"))
            y = (torch.nn.functional.gelu(h @ top(p + "mlp.gate").T, approximate="tanh") * (h @ top(p + "mlp.up").T)) @ top(p + "mlp.down").T
            x = x + _rms(y, top(p + "norm2b")) * top(p + "ls2")
        else:
            y, new = mix(x)
            x = x + cfg["residual_mult"] * _rms(y, 1.0 + top(p + "norm1"))
            y = (x @ top(p + "mlp.up").T).clamp(min=0).square() @ top(p + "mlp.down").T
            x = x + cfg["residual_mult"] * _rms(y, 1.0 + top(p + "norm2"))
        kept.append(new)
    return x, kept


def _hybrid_logits(cfg, weights, h):
    if cfg["architecture"] == "Latodra":
        return _rms(h, weights["final.norm"].double()) @ weights["embed"].double().T
    return _rms(h, 1.0 + weights["final.norm"].double()) @ weights["head"].double().T
