"""The attention calls whose speed matters, as a user of this package makes them.

A diffusion sampler calls the operator a few hundred times per step on image, video and prompt tokens; an LLM calls it
once per layer over the prompt and then once per layer and token over its cache.  Each case below is one such call
through the public Python surface on tensors that are already on the GPU, with the output allocated by the call unless
the program would keep it.  Sizes are those of the benchmark, the configurations and the tests of this repository, or
generic ones between them; inputs are N(0,1), as queries and keys behind a normalisation are.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "draw-things-community_b200"))
import dtattn  # noqa: E402

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # One token of an LLM with a short conversation behind it: query and key norms, rotary (a quarter of the
        # dimensions), cache append and attention, once per full-attention layer.  The smallest call: latency.
        dict(name="step_one_token_2k", kind="step", B=1, T=2048, Hq=16, Hkv=4, D=256, rot=64, norm=True, dtype="bf16"),
        # One token of an LLM of the other family (64 heads over one shared KV head of dim 512): a window of raw rows
        # and 512 selected rows of a compressed cache, with sinks.
        dict(name="sparse_step_8k", kind="sparse", Sq=1, Sr=8192, ratio=4, H=64, D=512, W=128, top=512, dtype="bf16"),
        # A batch of sixteen conversations at 8192 tokens: the cache streams from memory once per token and layer.
        dict(name="decode_batch16_8k", kind="decode", B=16, T=8192, Hq=32, Hkv=8, D=128, dtype="f16"),
        # Prompt tokens of an LLM text encoder: causal and padding mask together, a length as prompts have it.
        dict(name="encoder_masked_333", kind="masked", B=1, S=333, Hq=32, Hkv=8, D=128, causal=True, real=0.8, dtype="bf16"),
        # Text conditioning of a UNet at 1024 x 1024: 4096 image queries, both guidance branches, 77 prompt tokens.
        dict(name="cross_sdxl_77", kind="cross", B=2, Sq=4096, Sk=77, H=20, D=64, dtype="f16"),
        # Normalisation and rotary of queries and keys in front of the joint attention below.
        dict(name="prologue_joint_4608", kind="prologue", S=4608, H=24, D=128, per_token=False, dtype="bf16"),
        # UNet self-attention with the output projection that belongs to the node.
        dict(name="projected_self_4096", kind="projected", B=2, S=4096, H=20, D=64, C=1280, dtype="f16"),
        # A prompt read in chunks: 1777 new tokens behind 4096 cached ones, grouped heads of dim 256.
        dict(name="prefill_chunk_d256", kind="prefill", B=1, Sq=1777, Sk=5873, Hq=16, Hkv=4, D=256, dtype="bf16"),
        # UNet self-attention for models that must upcast it to 32 bits.
        dict(name="upcast_self_f32_4096", kind="self", B=2, S=4096, H=8, D=40, dtype="f32"),
        # Joint attention of image and text tokens in a diffusion transformer: the benchmark's own shape.
        dict(name="joint_4608", kind="self", B=1, S=4608, H=24, D=128, dtype="bf16"),
        # A prompt of 4096 tokens of the sparse-attention LLM.
        dict(name="sparse_prompt_4k", kind="sparse", Sq=4096, Sr=4096, ratio=4, H=64, D=512, W=128, top=512, dtype="bf16"),
        # Self-attention over the tokens of a 720p video clip: the largest call.
        dict(name="video_self_75600", kind="self", B=1, S=75600, H=40, D=128, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "sparse", "decode", "masked", "cross", "prologue", "projected", "prefill", "upcast", "self"])
    half = rng.choice(["f16", "bf16"])
    if kind in ("step", "decode"):
        Hq, Hkv, D = rng.choice([(16, 4, 256), (8, 2, 256), (32, 8, 128), (16, 8, 128), (32, 8, 64)])
        c = dict(kind=kind, B=rng.choice([1, 1, 2, 3, 4, 8, 16]), T=_log(rng, 64, 16384), Hq=Hq, Hkv=Hkv, D=D, dtype=half)
        if kind == "step":
            c.update(rot=D // rng.choice([1, 4]), norm=rng.random() < 0.5)
        return c
    if kind == "sparse":  # decode steps, a few tokens at a time, and prompts
        Sq = rng.choice([1, 1, 2, _log(rng, 3, 4096), _log(rng, 64, 4096)])
        past = _log(rng, 128, 12288) if Sq < 64 or rng.random() < 0.3 else 0
        return dict(kind=kind, Sq=Sq, Sr=Sq + past, ratio=4, H=64, D=512, W=128, top=rng.choice([256, 512]), dtype=half)
    if kind == "masked":  # CLIP-sized and LLM-sized text encoders
        if rng.random() < 0.3:
            return dict(kind=kind, B=rng.choice([1, 2]), S=77, Hq=12, Hkv=12, D=64, causal=True, real=1.0, dtype="f16")
        Hq, Hkv, D = rng.choice([(32, 8, 128), (16, 8, 256), (20, 20, 64)])
        return dict(kind=kind, B=rng.choice([1, 1, 2]), S=_log(rng, 40, 4096), Hq=Hq, Hkv=Hkv, D=D,
                    causal=rng.random() < 0.7, real=round(rng.uniform(0.3, 1.0), 3), dtype=half)
    if kind == "cross":
        if rng.random() < 0.7:  # UNets: heads of 40 or 64 over one or two prompts' worth of tokens
            D, H = rng.choice([(40, 8), (64, 10), (64, 20)])
            return dict(kind=kind, B=rng.choice([1, 2, 2, 4]), Sq=_log(rng, 256, 9216), Sk=rng.choice([77, 77, 154]), H=H, D=D, dtype="f16")
        return dict(kind=kind, B=1, Sq=_log(rng, 2048, 75600), Sk=rng.choice([257, 512]), H=rng.choice([12, 40]), D=128, dtype="bf16")
    if kind == "prologue":
        return dict(kind=kind, S=_log(rng, 256, 32768), H=rng.choice([5, 12, 24]), D=128, per_token=rng.random() < 0.4, dtype="bf16")
    if kind == "projected":
        H, D = rng.choice([(10, 64), (20, 64), (24, 128), (8, 40), (8, 80)])
        return dict(kind=kind, B=rng.choice([1, 2]), S=_log(rng, 256, 6144), H=H, D=D, C=H * D, dtype=half)
    if kind == "prefill":
        Hq, Hkv, D = rng.choice([(16, 4, 256), (32, 8, 128), (32, 8, 64)])
        Sq = _log(rng, 64, 8192)
        return dict(kind=kind, B=1, Sq=Sq, Sk=Sq + rng.choice([0, _log(rng, 64, 8192)]), Hq=Hq, Hkv=Hkv, D=D, dtype="bf16")
    if kind == "upcast":
        H, D = rng.choice([(8, 40), (5, 64), (10, 64), (8, 80)])
        return dict(kind="self", B=rng.choice([1, 2]), S=_log(rng, 256, 6144), H=H, D=D, dtype="f32")
    B, H, D, lo, hi, dt = rng.choice([
        (2, 8, 40, 256, 9216, "f16"), (2, 8, 80, 256, 2304, "f16"), (2, 8, 160, 64, 576, "f16"), (2, 10, 64, 256, 9216, "f16"),
        (2, 20, 64, 256, 4096, "f16"), (1, 24, 128, 512, 16384, "bf16"), (1, 12, 256, 512, 8192, "bf16"), (1, 12, 128, 4096, 32768, "bf16")])
    return dict(kind="self", B=B, S=_log(rng, lo, hi), H=H, D=D, dtype=dt)


def _operator(case, **kw):
    flags = [] if case["dtype"] == "f32" else [dtattn.GEMMFlag.Float16]
    return dtattn.ScaledDotProductAttention(scale=case["D"] ** -0.5, flags=flags, **kw)


def _rotary(g, tokens, D, rot, dtype, device):
    """Interleaved cos / sin per token; dimensions from `rot` on are not rotated."""
    angle = torch.rand(tokens, D // 2, generator=g, device=device) * (2 * math.pi)
    angle[:, rot // 2:] = 0
    return torch.stack([angle.cos(), angle.sin()], dim=-1).reshape(1, tokens, D).to(dtype)


def prepare(case, seed):
    dev, kind = torch.device("cuda"), case["kind"]
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=dev, dtype=torch.float32).to(dt)  # noqa: E731
    D, s = case["D"], dict(kind=kind)
    if kind == "self":
        shape = (case["B"], case["S"], case["H"], D)
        s.update(op=_operator(case), q=rnd(*shape), k=rnd(*shape), v=rnd(*shape))
    elif kind == "cross":
        B, H = case["B"], case["H"]
        s.update(op=_operator(case), q=rnd(B, case["Sq"], H, D), k=rnd(B, case["Sk"], H, D), v=rnd(B, case["Sk"], H, D))
    elif kind == "prefill":
        B, Sk, Hkv = case["B"], case["Sk"], case["Hkv"]
        s.update(op=_operator(case, is_causal=True), q=rnd(B, case["Sq"], case["Hq"], D), k=rnd(B, Sk, Hkv, D), v=rnd(B, Sk, Hkv, D))
    elif kind == "masked":
        B, S, Hkv = case["B"], case["S"], case["Hkv"]
        mask = torch.zeros(1, 1, S, S, device=dev, dtype=dt)
        real = max(1, round(S * case["real"]))  # the positions behind the prompt are padding
        mask[..., real:] = -torch.finfo(dt).max
        s.update(op=_operator(case, is_causal=case["causal"], has_attention_mask=True), q=rnd(B, S, case["Hq"], D),
                 k=rnd(B, S, Hkv, D), v=rnd(B, S, Hkv, D), mask=mask)
        if not case["causal"] and real < S:
            s["mask"][..., real:, :real] = -torch.finfo(dt).max  # padding attends to padding only, the prompt to itself
            s["mask"][..., real:, real:] = 0
    elif kind == "projected":
        B, S, H, C = case["B"], case["S"], case["H"], case["C"]
        op = _operator(case, multi_head_output_projection_fused=True)
        op.set_output_projection(rnd(C, H * D) * (H * D) ** -0.5, rnd(C))
        s.update(op=op, q=rnd(B, S, H, D), k=rnd(B, S, H, D), v=rnd(B, S, H, D))
    elif kind == "decode":
        B, T, Hkv = case["B"], case["T"], case["Hkv"]
        s.update(op=_operator(case, is_causal=True), q=rnd(B, 1, case["Hq"], D), k=rnd(B, T, Hkv, D), v=rnd(B, T, Hkv, D))
    elif kind == "step":
        B, T, Hkv = case["B"], case["T"], case["Hkv"]
        s.update(scale=D ** -0.5, cached=T - 1, q=rnd(B, 1, case["Hq"], D), k_new=rnd(B, 1, Hkv, D), v_new=rnd(B, 1, Hkv, D),
                 k_cache=rnd(B, T, Hkv, D), v_cache=rnd(B, T, Hkv, D), rotary=_rotary(g, 1, D, case["rot"], dt, dev),
                 q_norm_weight=rnd(D) if case["norm"] else None, k_norm_weight=rnd(D) if case["norm"] else None)
    elif kind == "prologue":
        S, H = case["S"], case["H"]
        n = H * D if case["per_token"] else D
        s.update(q=rnd(1, S, H, D), k=rnd(1, S, H, D), q_weight=rnd(n), k_weight=rnd(n), per_token=case["per_token"],
                 rotary=_rotary(g, S, D, D, dt, dev).view(1, S, 1, D), post_scale=D ** -0.25 if case["per_token"] else 1.0)
    elif kind == "sparse":
        Sq, Sr = case["Sq"], case["Sr"]
        Sc = Sr // case["ratio"]  # one compressed row per `ratio` raw rows
        q, raw, comp, sinks = rnd(1, Sq, case["H"], D), rnd(1, Sr, 1, D), rnd(1, Sc, 1, D), rnd(case["H"])
        # the indexer's choice: a token's best rows among those whose raw rows all lie at or before it, -1 where there
        # are fewer than asked for
        seen = (torch.arange(Sr - Sq, Sr, device=dev) + 1) // case["ratio"]
        score = torch.rand(Sq, Sc, generator=g, device=dev).masked_fill(torch.arange(Sc, device=dev) >= seen[:, None], -1.0)
        best = score.topk(min(case["top"], Sc), dim=-1)
        selected = torch.where(best.values < 0, -1, best.indices).to(torch.int32)
        s.update(op=dtattn.SparseIndexedAttention(scale=D ** -0.5, sliding_window=case["W"]), q=q, raw=raw, comp=comp,
                 selected=selected, sinks=sinks.view(1, 1, -1, 1))
    return s


def run(s):
    kind = s["kind"]
    if kind == "masked":
        return s["op"](s["q"], s["k"], s["v"], s["mask"])
    if kind == "step":
        out = dtattn.decode_step(s["q"], s["k_cache"], s["v_cache"], s["k_new"], s["v_new"], s["rotary"], s["scale"], s["cached"],
                                 q_norm_weight=s["q_norm_weight"], k_norm_weight=s["k_norm_weight"])
        return {"out": out, "k_cache": s["k_cache"], "v_cache": s["v_cache"]}
    if kind == "prologue":
        return dtattn.qk_prologue(s["q"], s["k"], q_weight=s["q_weight"], k_weight=s["k_weight"], rotary=s["rotary"],
                                  norm_per_token=s["per_token"], post_scale=s["post_scale"])
    if kind == "sparse":
        return s["op"](s["q"], s["raw"], s["raw"], s["comp"], s["comp"], s["selected"], s["sinks"])
    return s["op"](s["q"], s["k"], s["v"])


def _attend(q, k, v, scale, visible=None, bias=None):
    """softmax(scale Q K^T + bias) V in 64 bits, one (image, KV head) and a run of query rows at a time."""
    B, Sq, Hq, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    out = torch.empty(B, Sq, Hq, D, dtype=torch.float64, device=q.device)
    rows = max(1, min(Sq, (1 << 27) // (Sk * (Hq // Hkv))))
    for b in range(B):
        for h in range(Hkv):
            heads = slice(h * (Hq // Hkv), (h + 1) * (Hq // Hkv))
            kt, vv = k[b, :, h].double().t().contiguous(), v[b, :, h].double()
            for r in range(0, Sq, rows):
                s = torch.matmul(q[b, r:r + rows, heads].double().transpose(0, 1), kt).mul_(scale)  # [heads, rows, Sk]
                if bias is not None:
                    s += bias[r:r + rows].double()
                if visible is not None:
                    i = torch.arange(r, r + s.shape[1], device=q.device)[:, None]
                    s.masked_fill_(~visible(i, torch.arange(Sk, device=q.device)), -math.inf)
                out[b, r:r + rows, heads] = torch.matmul(torch.softmax(s, dim=-1), vv).transpose(0, 1)
    return out


def _rotate(x, table):
    """Pairs of dimensions as complex numbers times cos + i sin."""
    x, t = x.unflatten(-1, (-1, 2)), table.double().unflatten(-1, (-1, 2))
    re = x[..., 0] * t[..., 0] - x[..., 1] * t[..., 1]
    im = x[..., 0] * t[..., 1] + x[..., 1] * t[..., 0]
    return torch.stack([re, im], dim=-1).flatten(-2)


def _rms(x, weight, dims):
    return x if weight is None else x * torch.rsqrt((x * x).mean(dim=dims, keepdim=True) + 1e-6) * weight.double()


def exact(case, seed):
    """What `run` returns, in 64 bits from the same inputs."""
    if work(case)["flops"] > 3e13:  # the 720p clip: minutes of 64-bit arithmetic
        return None
    s, kind, D = prepare(case, seed), case["kind"], case["D"]
    if kind in ("self", "cross"):
        return _attend(s["q"], s["k"], s["v"], D ** -0.5)
    if kind in ("prefill", "decode"):
        past = s["k"].shape[1] - s["q"].shape[1]
        return _attend(s["q"], s["k"], s["v"], D ** -0.5, lambda i, j: j <= i + past)
    if kind == "masked":
        return _attend(s["q"], s["k"], s["v"], D ** -0.5, (lambda i, j: j <= i) if case["causal"] else None, s["mask"][0, 0])
    if kind == "projected":
        op = s["op"]
        return _attend(s["q"], s["k"], s["v"], D ** -0.5).flatten(2) @ op.weight.double().t() + op.bias.double()
    if kind == "step":
        table = s["rotary"].view(1, 1, 1, D)
        q = _rotate(_rms(s["q"].double(), s["q_norm_weight"], -1), table)
        k, v = s["k_cache"].double(), s["v_cache"].double()
        k[:, s["cached"]:] = _rotate(_rms(s["k_new"].double(), s["k_norm_weight"], -1), table)
        v[:, s["cached"]:] = s["v_new"].double()
        return {"out": _attend(q, k, v, D ** -0.5), "k_cache": k, "v_cache": v}
    if kind == "prologue":
        outs = []
        for x, w in ((s["q"], s["q_weight"]), (s["k"], s["k_weight"])):
            n = _rms(x.double().flatten(2), w, -1).view(x.shape) if s["per_token"] else _rms(x.double(), w, -1)
            outs.append(_rotate(n, s["rotary"]) * s["post_scale"])
        return tuple(outs)
    q, raw, comp, selected = s["q"][0].double(), s["raw"][0, :, 0].double(), s["comp"][0, :, 0].double(), s["selected"].long()
    Sq, Sr, W = case["Sq"], case["Sr"], case["W"]
    out, sinks = torch.empty_like(q), s["sinks"].double().reshape(-1, 1)
    for r in range(0, Sq, 128):
        own = torch.arange(Sr - Sq + r, Sr - Sq + min(Sq, r + 128), device=q.device)[:, None]
        near = own - torch.arange(min(W, Sr), device=q.device)
        picked = selected[r:r + 128]
        keys = torch.cat([raw[near.clamp(min=0)], comp[picked.clamp(min=0)]], dim=1)  # [tokens, keys, D]
        score = torch.matmul(q[r:r + 128], keys.transpose(1, 2)).mul_(D ** -0.5)  # [tokens, heads, keys]
        score.masked_fill_(torch.cat([near, picked], dim=1)[:, None] < 0, -math.inf)
        p = torch.softmax(torch.cat([score, sinks.expand(score.shape[0], -1, 1)], dim=-1), dim=-1)[..., :-1]
        out[r:r + 128] = torch.matmul(p, keys)
    return out[None]


def work(case):
    """Visible (query, key) pairs count, four FLOPs per pair and dimension; every tensor moves once."""
    kind, D, es = case["kind"], case["D"], 4 if case["dtype"] == "f32" else 2
    if kind == "self":
        n = case["B"] * case["S"] * case["H"] * D
        return {"bytes": es * 4 * n, "flops": 4 * n * case["S"]}
    if kind == "cross":
        n = case["B"] * case["H"] * D
        return {"bytes": es * n * 2 * (case["Sq"] + case["Sk"]), "flops": 4 * n * case["Sq"] * case["Sk"]}
    if kind == "prefill":
        B, Sq, Sk = case["B"], case["Sq"], case["Sk"]
        pairs = Sq * (Sk - Sq) + Sq * (Sq + 1) // 2
        return {"bytes": es * B * D * 2 * (Sq * case["Hq"] + Sk * case["Hkv"]), "flops": 4 * B * case["Hq"] * D * pairs}
    if kind == "masked":
        B, S = case["B"], case["S"]
        real = max(1, round(S * case["real"]))
        if case["causal"]:
            pairs = real * (real + 1) // 2 + (S - real) * real
        else:
            pairs = real * real + (S - real) ** 2
        return {"bytes": es * (B * S * D * 2 * (case["Hq"] + case["Hkv"]) + S * S), "flops": 4 * B * case["Hq"] * D * pairs}
    if kind == "projected":
        rows, n, C = case["B"] * case["S"], case["H"] * D, case["C"]
        return {"bytes": es * (rows * (3 * n + C) + n * C), "flops": 4 * rows * n * case["S"] + 2 * rows * n * C}
    if kind in ("decode", "step"):
        B, T, Hq, Hkv = case["B"], case["T"], case["Hq"], case["Hkv"]
        moved = 2 * T * Hkv * D + 2 * Hq * D + (2 * Hkv * D if kind == "step" else 0)
        return {"bytes": es * B * moved, "flops": 4 * B * Hq * T * D}
    if kind == "prologue":
        n = case["S"] * case["H"] * D
        return {"bytes": es * (4 * n + case["S"] * D), "flops": 10 * 2 * n}
    Sq, Sr, H, ratio, W = case["Sq"], case["Sr"], case["H"], case["ratio"], case["W"]
    Sc = Sr // ratio
    keys, picked = 0, 0
    for i in range(Sr - Sq, Sr):
        n = min(case["top"], Sc, (i + 1) // ratio)
        picked += n
        keys += min(W, i + 1) + n
    rows = min(Sr, Sq + W - 1) + min(Sc, picked)
    return {"bytes": es * D * (2 * Sq * H + rows) + 4 * Sq * min(case["top"], Sc), "flops": 4 * H * D * keys}


def tolerance(case):
    """About four times the largest distance from the same path in 64 bits that was measured over these ranges: 3.6e-4
    for f16 and 2.9e-3 for bf16 (a 16-bit result and 16-bit softmax weights), 1.4e-6 for f32 (sums over the keys)."""
    return {"rel": {"f32": 6e-6, "f16": 1.5e-3, "bf16": 1.2e-2}[case["dtype"]]}
