"""The performance cases of this library: what a program that trains or serves a GPT-2 style model asks of it, called the
way such a program calls it.

A case is a plain dict; `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges, `prepare(case, seed)` what
the program holds before the call (tensors on the GPU, buffers that it keeps from step to step, tables built once),
`run(state)` one pass through the public entry points, `work(case)` the bytes and operations that pass cannot do without and
`tolerance(case)` how far two correct implementations may lie apart.

Kinds of case:
  attention     the attention op alone: forward, or forward and backward of a training step (fp32 API and bf16 variant)
  context       the same through AttentionContext, the object that the static engine holds per layer (batch 1, legacy symbols)
  token         one generated token through a whole layer, reading and extending a contiguous fp32 cache
  paged_decode  one token's attention over a long paged cache
  layer         everything of a layer's step around attention: LayerNorm, projections, GELU, forward and backward forms
  adamw         the optimizer's step over all parameter tensors of a model
  loss          softmax and cross-entropy of one chunk of logits
"""
import math

import torch

from __graft_entry__ import load_package

df = load_package()

# GPT-2 small, the model of this repository's full-step benchmark
WIDTH, HEADS, HEAD_DIM, FF, LAYERS, VOCAB, POSITIONS = 768, 12, 64, 3072, 12, 50257, 4096


def _attention(name, dtype, direction, batch, heads, seq, head_dim, causal=True):
    c = {"kind": "attention", "dtype": dtype, "direction": direction, "batch": batch, "heads": heads, "seq": seq,
         "head_dim": head_dim, "causal": causal}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest configuration that the benchmark names: one short sequence. Launches and host work are what count.
        _attention("train_b1_s128", "fp32", "train", 1, HEADS, 128, HEAD_DIM),
        # The headline configuration: the attention of one GPT-2 small layer in a training step.
        _attention("train_b8_s1024", "fp32", "train", 8, HEADS, 1024, HEAD_DIM),
        # A long training sequence: the forward and backward of bench_sequence_limit's lower end.
        _attention("train_b1_s8192", "fp32", "train", 1, HEADS, 8192, HEAD_DIM),
        # Prefill of a long prompt: forward only, where the sequence-limit sweep is quoted.
        _attention("prefill_s32768", "fp32", "forward", 1, HEADS, 32768, HEAD_DIM),
        # The bf16 variant with the head size of the long-context ring configuration.
        _attention("train_bf16_d128_s8192", "bf16", "train", 1, 16, 8192, 128),
        # The fp32 API with a head size other than 64 (any up to 128 is taken), ragged length, full fp32 arithmetic.
        _attention("train_d128_s1000", "fp32", "train", 2, 8, 1000, 128),
        # The static engine's call per layer: one ragged sequence, no saved output, caller-owned scratch.
        {"name": "context_s1531", "kind": "context", "heads": HEADS, "seq": 1531, "head_dim": HEAD_DIM, "causal": True},
        # Generating text: one token through a layer with a few hundred tokens in the cache.
        {"name": "token_t300", "kind": "token", "heads": HEADS, "head_dim": HEAD_DIM, "ff": FF, "cached": 300},
        # One token over a long bf16 paged cache, pages of 16 tokens, no scratch lent.
        {"name": "paged_bf16_t65537", "kind": "paged_decode", "heads": 16, "head_dim": 128, "tokens": 65537, "page": 16,
         "dtype": "bf16", "scratch": False},
        # The rest of a layer in a training step: batch 8 of 1024 tokens.
        {"name": "layer_rows8192", "kind": "layer", "rows": 8192, "width": WIDTH, "ff": FF},
        # The optimizer step of GPT-2 small: 124 M parameters in 196 tensors.
        {"name": "adamw_gpt2_small", "kind": "adamw", "layers": LAYERS, "width": WIDTH, "vocab": VOCAB, "positions": 1024},
        # The loss head's chunk of the training step: 512 rows of the GPT-2 vocabulary (odd row length).
        {"name": "loss_512x50257", "kind": "loss", "rows": 512, "vocab": VOCAB, "train": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("fp32", "fp32", "prefill", "bf16", "head", "context", "token", "paged_decode", "layer", "adamw", "loss"))
    causal = rng.random() < 0.85
    if kind == "fp32":  # training sequences from a short sentence to 8K, batches that keep the tokens of a step bounded
        seq = _log(rng, 32, 8192)
        return _attention(None, "fp32", "train", rng.randint(1, max(1, min(8, 8192 // seq))), rng.choice((4, 8, 12, 16)) if seq < 6000 else 8, seq,
                          HEAD_DIM, causal)
    if kind == "prefill":
        return _attention(None, "fp32", "forward", 1, rng.choice((4, 8, 12)), _log(rng, 128, 30000), HEAD_DIM, True)
    if kind == "bf16":
        seq = _log(rng, 128, 8192)
        return _attention(None, "bf16", "train", rng.randint(1, max(1, min(8, 8192 // seq))), rng.choice((8, 12, 16)), seq, rng.choice((64, 128)), causal)
    if kind == "head":
        seq = _log(rng, 64, 1400)
        return _attention(None, "fp32", "train", 1 if seq > 1000 else rng.randint(1, 2), rng.choice((4, 6, 8)), seq, rng.choice((32, 48, 80, 96, 128)), causal)
    if kind == "context":
        return {"kind": "context", "heads": rng.choice((1, 8, 12)), "seq": _log(rng, 64, 4096), "head_dim": HEAD_DIM, "causal": causal}
    if kind == "token":
        heads = rng.choice((8, 12, 16))
        return {"kind": "token", "heads": heads, "head_dim": HEAD_DIM, "ff": 4 * heads * HEAD_DIM, "cached": _log(rng, 16, 4096)}
    if kind == "paged_decode":
        d = rng.choice((64, 128))
        return {"kind": "paged_decode", "heads": rng.choice((8, 12, 16)), "head_dim": d, "tokens": _log(rng, 500, 130000 if d == 64 else 65000),
                "page": rng.choice((16, 32)), "dtype": rng.choice(("fp32", "bf16")), "scratch": rng.random() < 0.4}
    if kind == "layer":
        width = rng.choice((512, 768, 1024))
        return {"kind": "layer", "rows": _log(rng, 100, 8192 * 768 // width), "width": width, "ff": 4 * width}
    if kind == "adamw":
        width = rng.choice((256, 384, 512, 768))
        return {"kind": "adamw", "layers": rng.randint(2, 12), "width": width, "vocab": _log(rng, 5000, VOCAB), "positions": rng.choice((256, 512, 1024))}
    return {"kind": "loss", "rows": _log(rng, 32, 512), "vocab": _log(rng, 5000, VOCAB), "train": rng.random() < 0.7}


class _Normal:
    """Seeded normal tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def __call__(self, *shape, std=1.0, dtype=torch.float32):
        x = torch.randn(shape, generator=self.gen, device="cuda", dtype=torch.float32)
        return (x if std == 1.0 else x.mul_(std)).to(dtype)


def _empty_like(*tensors):
    return [torch.empty_like(t) for t in tensors]


def prepare(case, seed):
    n = _Normal(seed)
    s = dict(case)
    kind = case["kind"]
    if kind == "attention":
        B, H, S, D = case["batch"], case["heads"], case["seq"], case["head_dim"]
        dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        s["q"], s["k"], s["v"], s["d_out"] = (n(B, S, H * D, dtype=dt) for _ in range(4))
        s["out"], s["d_q"], s["d_k"], s["d_v"] = _empty_like(s["q"], s["q"], s["q"], s["q"])
        s["lse"], s["delta"] = (torch.empty((B, H, S), device="cuda") for _ in range(2))
        s["scale"] = D ** -0.5
    elif kind == "context":
        H, S, D = case["heads"], case["seq"], case["head_dim"]
        s["q"], s["k"], s["v"], s["d_out"] = (n(S, H * D) for _ in range(4))
        s["out"], s["d_q"], s["d_k"], s["d_v"] = _empty_like(s["q"], s["q"], s["q"], s["q"])
        # the scratch that all layers of an engine share, of the size that the backward asks for
        s["context"] = df.AttentionContext.new_shared(H, S, D, [torch.empty(H * 2 * S * S, device="cuda")])
        s["scale"] = D ** -0.5
    elif kind == "token":
        H, D, T, ff = case["heads"], case["head_dim"], case["cached"], case["ff"]
        w = H * D
        s["x"] = n(1, w)
        s["gamma"], s["beta"] = [1.0 + n(w, std=0.02) for _ in range(2)], [n(w, std=0.02) for _ in range(2)]
        s["w"] = [n(w, w, std=0.02) for _ in range(4)] + [n(ff, w, std=0.02), n(w, ff, std=0.02)]
        s["b"] = [n(w, std=0.02) for _ in range(4)] + [n(ff, std=0.02), n(w, std=0.02)]
        s["k_cache"], s["v_cache"] = n(POSITIONS + 1, w), n(POSITIONS + 1, w)
        s["row"] = torch.empty((7, w), device="cuda")
        s["act"], s["stat"] = torch.empty((1, ff), device="cuda"), torch.empty((4, 1), device="cuda")
        s["scale"] = D ** -0.5
    elif kind == "paged_decode":
        H, D, T, page = case["heads"], case["head_dim"], case["tokens"], case["page"]
        dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        pages = (T + page - 1) // page
        s["q"] = n(H * D)
        s["k_pool"], s["v_pool"] = (n(pages * page, H * D, dtype=dt) for _ in range(2))
        s["table"] = torch.randperm(pages, generator=n.gen, device="cuda").to(torch.int32)
        s["out"] = torch.empty(H * D, device="cuda")
        s["max_chunks"] = (T + 255) // 256 if case["scratch"] else 0
        s["partials"] = tuple(torch.empty(H * s["max_chunks"] * m, device="cuda") for m in (1, 1, D)) if case["scratch"] else None
        s["scale"] = D ** -0.5
    elif kind == "layer":
        rows, w, ff = case["rows"], case["width"], case["ff"]
        s["x"], s["attended"], s["d_act"], s["d_norm"] = n(rows, w), n(rows, w), n(rows, ff), n(rows, w)
        s["gamma"], s["beta"] = [1.0 + n(w, std=0.02) for _ in range(2)], [n(w, std=0.02) for _ in range(2)]
        s["w"] = [n(w, w, std=0.02) for _ in range(4)] + [n(ff, w, std=0.02), n(w, ff, std=0.02)]
        s["b"] = [n(w, std=0.02) for _ in range(4)] + [n(ff, std=0.02), n(w, std=0.02)]
        s["h1"], s["q"], s["k"], s["v"], s["x1"], s["h2"], s["x2"], s["d_x"] = _empty_like(*[s["x"]] * 8)
        s["pre"], s["act"], s["d_pre"] = _empty_like(*[s["d_act"]] * 3)
        s["stat"] = torch.empty((4, rows), device="cuda")
        s["d_gamma"], s["d_beta"] = torch.zeros(w, device="cuda"), torch.zeros(w, device="cuda")
    elif kind == "adamw":
        sizes = _parameter_sizes(case)
        offsets, total = [], 0
        for m in sizes:  # one arena, every tensor on a 256-byte boundary
            offsets.append(total)
            total += (m + 63) // 64 * 64
        s["p"], s["m"], s["g"] = n(total, std=0.02), n(total, std=1e-3), n(total, std=1e-3)
        s["v"] = n(total, std=1e-3).square_()
        s["plan"] = df.AdamwPlan([tuple(s[a][o:o + m] for a in "pmvg") for o, m in zip(offsets, sizes)])
    else:
        rows, vocab = case["rows"], case["vocab"]
        s["logits"] = n(rows, vocab, std=2.0)
        s["targets"] = torch.randint(0, vocab, (rows,), generator=n.gen, device="cuda", dtype=torch.int32)
        s["grad"] = torch.empty_like(s["logits"]) if case["train"] else None
        s["loss"] = torch.zeros(1, device="cuda")
    return s


def _parameter_sizes(case):
    w = case["width"]
    block = [w, w] + [w * w, w] * 4 + [w, w] + [4 * w * w, 4 * w, 4 * w * w, w]
    return [case["vocab"] * w, case["positions"] * w] + block * case["layers"] + [w, w]


def run(s):
    kind = s["kind"]
    if kind == "attention":
        q, k, v, out, lse, heads, scale, causal = s["q"], s["k"], s["v"], s["out"], s["lse"], s["heads"], s["scale"], s["causal"]
        bf16 = s["dtype"] == "bf16"
        (df.forward_bf16 if bf16 else df.forward)(q, k, v, heads, scale, causal, out=out, lse=lse)
        if s["direction"] == "forward":
            return out, lse
        (df.backward_bf16 if bf16 else df.backward)(q, k, v, out, s["d_out"], lse, heads, scale, causal, d_q=s["d_q"], d_k=s["d_k"],
                                                    d_v=s["d_v"], delta_buf=s["delta"])
        return out, lse, s["d_q"], s["d_k"], s["d_v"]
    if kind == "context":
        c = s["context"]
        c.forward_device_into(s["q"], s["k"], s["v"], s["scale"], s["causal"], s["out"])
        c.backward_device_into(s["q"], s["k"], s["v"], s["d_out"], s["scale"], s["causal"], s["d_q"], s["d_k"], s["d_v"])
        return s["out"], s["d_q"], s["d_k"], s["d_v"]
    if kind == "token":
        t, row, stat, w, b = s["cached"], s["row"], s["stat"], s["w"], s["b"]
        h1, q, a, x1, h2, x2 = (row[i:i + 1] for i in range(6))
        k, v = s["k_cache"][t:t + 1], s["v_cache"][t:t + 1]
        df.layernorm(s["x"], s["gamma"][0], s["beta"][0], out=h1, means=stat[0], rstds=stat[1])
        df.linear_qkv(h1, w[0], w[1], w[2], b[0], b[1], b[2], q=q, k=k, v=v)
        df.decode(q, s["k_cache"], s["v_cache"], s["heads"], t + 1, s["scale"], out=a)
        df.linear(a, w[3], b[3], residual=s["x"], out=x1)
        df.layernorm(x1, s["gamma"][1], s["beta"][1], out=h2, means=stat[2], rstds=stat[3])
        df.linear_gelu(h2, w[4], b[4], out=s["act"], keep_pre_activation=False)
        df.linear(s["act"], w[5], b[5], residual=x1, out=x2)
        return q, k, v, a, x1, s["act"], x2
    if kind == "paged_decode":
        return df.decode(s["q"], s["k_pool"], s["v_pool"], s["heads"], s["tokens"], s["scale"], block_table=s["table"], page_size=s["page"],
                         partials=s["partials"], max_chunks=s["max_chunks"], out=s["out"])
    if kind == "layer":
        w, b, stat = s["w"], s["b"], s["stat"]
        df.layernorm(s["x"], s["gamma"][0], s["beta"][0], out=s["h1"], means=stat[0], rstds=stat[1])
        df.linear_qkv(s["h1"], w[0], w[1], w[2], b[0], b[1], b[2], q=s["q"], k=s["k"], v=s["v"])
        df.linear(s["attended"], w[3], b[3], residual=s["x"], out=s["x1"])
        df.layernorm(s["x1"], s["gamma"][1], s["beta"][1], out=s["h2"], means=stat[2], rstds=stat[3])
        df.linear_gelu(s["h2"], w[4], b[4], pre_activation=s["pre"], out=s["act"])
        df.linear(s["act"], w[5], b[5], residual=s["x1"], out=s["x2"])
        df.gelu_backward(s["d_act"], s["pre"], grad_x=s["d_pre"])
        # the weight gradients add up over the micro-batches of a step
        df.layernorm_backward(s["d_norm"], s["x1"], s["gamma"][1], stat[2], stat[3], grad_x=s["d_x"], grad_gamma=s["d_gamma"], grad_beta=s["d_beta"])
        return {a: s[a] for a in ("h1", "q", "k", "v", "x1", "h2", "pre", "act", "x2", "d_pre", "d_x", "d_gamma", "d_beta", "stat")}
    if kind == "adamw":
        s["plan"].step(3e-4, 0.9, 0.95, 1e-8, 0.1, 1.0 - 0.9 ** 10, 1.0 - 0.95 ** 10)
        return s["p"], s["m"], s["v"]
    df.chunked_logit_ce(s["logits"], s["targets"], s["loss"], s["rows"], grad_logits=s["grad"])
    return (s["logits"], s["grad"], s["loss"]) if s["train"] else s["loss"]


def work(case):
    kind = case["kind"]
    if kind in ("attention", "context"):
        B, H, S, D = case.get("batch", 1), case["heads"], case["seq"], case["head_dim"]
        size = 2 if case.get("dtype") == "bf16" else 4
        train = case.get("direction", "train") == "train"
        one = B * S * H * D * size
        # products over the visible pairs: 2 in the forward; S again, dP, dV, dK and dQ in the backward
        pairs = S * (S + 1) // 2 if case["causal"] else S * S
        return {"bytes": (8 if train else 4) * one + B * H * S * 4, "flops": (7 if train else 2) * 2 * B * H * pairs * D}
    if kind == "token":
        w, ff, t = case["heads"] * case["head_dim"], case["ff"], case["cached"] + 1
        weights = 4 * w * w + 2 * w * ff
        return {"bytes": 4 * (weights + 2 * t * w + 13 * w + 2 * ff), "flops": 2 * weights + 4 * t * w}
    if kind == "paged_decode":
        w, t = case["heads"] * case["head_dim"], case["tokens"]
        return {"bytes": 2 * t * w * (2 if case["dtype"] == "bf16" else 4) + 8 * w + 4 * (t // case["page"]), "flops": 4 * t * w}
    if kind == "layer":
        rows, w, ff = case["rows"], case["width"], case["ff"]
        weights = 4 * w * w + 2 * w * ff
        # in: x, attended, d_norm, d_act; out: the two norms, q, k, v, x1, x2, d_x, pre, act, d_pre
        return {"bytes": 4 * (rows * (11 * w + 4 * ff) + weights), "flops": 2 * rows * weights}
    if kind == "adamw":
        n = sum(_parameter_sizes(case))
        return {"bytes": 28 * n, "flops": 15 * n}
    n = case["rows"] * case["vocab"]
    return {"bytes": (12 if case["train"] else 4) * n, "flops": 5 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "attention" and case["dtype"] == "bf16":
        return {"rel": 1e-2}
    if kind in ("layer", "token") or kind in ("attention", "context") and case["head_dim"] == HEAD_DIM:
        return {"rel": 2e-3}  # TF32 products (an 11-bit significand) with fp32 sums
    if kind == "adamw":
        return {"rel": 2e-6}  # element by element in fp32
    return {"rel": 1e-5}  # fp32 throughout
