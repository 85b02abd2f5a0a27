"""The workloads this package's speed is judged by: the quantized operators and the resident decoder,
called as a user's program calls them.

    listed()            the workloads, by name
    draw(rng)           another one of the same ranges
    prepare(case, seed) what the program holds before the call, on the GPU: inputs, packed weights, workspaces
    run(state)          one pass through the public entry points, and its outputs
    work(case)          bytes and operations that a pass cannot do without
    tolerance(case)     how far two correct implementations of the same precision may be apart

The kinds of work:

    int8     full-integer FULLY_CONNECTED (int8 in, int32 accumulate, requantized int8 out)
    hybrid   dynamic-range FULLY_CONNECTED (float rows quantized on the fly, int8 weights)
    int4     FULLY_CONNECTED over blockwise int4 weights with fp16 block scales
    sdpa     attention of one new token per sequence over its cached keys and values
    decode   a few tokens of greedy decoding of the Gemma-2B-shaped decoder, for a batch of sequences
    prefill  the prompt pass of one sequence, and the first step behind it
"""
import math

import numpy as np
import torch

from litert_b200 import decoder as dec
from litert_b200 import ops

# (query heads, KV heads, head size) that decoder models have: one shared KV head, groups of 2 to 8, one each
HEAD_LAYOUTS = ((8, 1, 256), (4, 1, 256), (8, 1, 128), (8, 2, 128), (16, 2, 128), (8, 4, 64), (8, 8, 64))


def listed():
    return [
        # a full-integer layer of a small network at an ordinary batch: everything is in L2, latency counts
        dict(name="int8 m32 2048x2048", op="int8", m=32, n=2048, k=2048, per_channel=True),
        # the smallest calls, nothing a multiple of anything: the classifier head of a small model
        dict(name="hybrid m3 500x300 bias relu6", op="hybrid", m=3, n=500, k=300, bias=True, activation=ops.ACT_RELU6,
             asymmetric=True),
        # the hidden -> feed-forward projection for one token and for a prompt chunk
        dict(name="hybrid m1 14336x4096", op="hybrid", m=1, n=14336, k=4096, bias=False, activation=ops.ACT_NONE,
             asymmetric=True),
        dict(name="hybrid m512 14336x4096", op="hybrid", m=512, n=14336, k=4096, bias=False, activation=ops.ACT_NONE,
             asymmetric=True),
        # the same for 4-bit weights
        dict(name="int4 m1 16384x2048", op="int4", m=1, n=16384, k=2048, block=32),
        dict(name="int4 m512 16384x2048", op="int4", m=512, n=16384, k=2048, block=32),
        # a serving batch of long, ragged sequences: fp16 cache and int8 cache with a scale per token
        dict(name="sdpa f16 16 x 8192", op="sdpa", b=16, n=8, nkv=1, h=256, s_max=8192, kv="f16", cap=0.0),
        dict(name="sdpa int8 16 x 8192", op="sdpa", b=16, n=8, nkv=1, h=256, s_max=8192, kv="i8", cap=0.0),
        # the composite as a graph holds it: float32 tensors, an additive mask over the whole cache, a logit cap
        dict(name="sdpa f32 mask 4 x 2000", op="sdpa", b=4, n=8, nkv=2, h=128, s_max=2000, kv="f32", cap=50.0),
        # an interactive reply and a full serving batch, both behind prompts of 1024 tokens
        dict(name="decode batch 1", op="decode", batch=1, context=1024, kv="f16", ragged=False),
        dict(name="decode batch 32", op="decode", batch=32, context=1024, kv="f16", ragged=False),
        # the prompt of an interactive request
        dict(name="prefill 1024", op="prefill", tokens=1024, kv="f16"),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A layer width: a multiple of 64 two times out of three, else anything."""
    v = _log(rng, lo, hi)
    return v if rng.random() < 1 / 3 else max(64, v // 64 * 64)


def draw(rng):
    op = rng.choice(("int8", "hybrid", "hybrid", "int4", "int4", "sdpa", "sdpa", "sdpa", "decode", "prefill"))
    if op == "int8":
        return dict(op=op, m=_log(rng, 1, 1024), n=_width(rng, 128, 8192), k=_width(rng, 128, 8192),
                    per_channel=rng.random() < 0.7)
    if op == "hybrid":
        return dict(op=op, m=_log(rng, 1, 512), n=_width(rng, 128, 14336), k=_width(rng, 128, 8192),
                    bias=rng.random() < 0.5, activation=rng.choice((ops.ACT_NONE, ops.ACT_NONE, ops.ACT_RELU, ops.ACT_RELU6)),
                    asymmetric=rng.random() < 0.8)
    if op == "int4":
        block = rng.choice((32, 32, 64, 128))
        return dict(op=op, m=_log(rng, 1, 512), n=_width(rng, 128, 16384), k=max(256, _log(rng, 256, 8192) // block * block),
                    block=block)
    if op == "sdpa":
        n, nkv, h = rng.choice(HEAD_LAYOUTS)
        kv = rng.choice(("f16", "f16", "i8", "f32"))
        s_max = _log(rng, 64, 8192)
        # no more cache than the largest listed case holds
        most = 16 * 8192 * 256 // (s_max * nkv * h * (2 if kv == "f32" else 1))
        return dict(op=op, b=_log(rng, 1, max(1, min(16, most))), n=n, nkv=nkv, h=h, s_max=s_max, kv=kv,
                    cap=rng.choice((0.0, 0.0, 50.0)))
    if op == "decode":
        return dict(op=op, batch=_log(rng, 1, 32), context=_log(rng, 16, 1024), kv=rng.choice(("f16", "i8")),
                    ragged=rng.random() < 0.5)
    return dict(op=op, tokens=_log(rng, 16, 1024), kv=rng.choice(("f16", "i8")))


# ---- inputs --------------------------------------------------------------------------------------------

#: Tokens of one decode pass.
REPLY = 16


def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _uniform(g, lo, hi, *shape):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _int8_weights(g, n, k):
    return _normal(g, n, k).mul_(40).round_().clamp_(-127, 127).to(torch.int8)


def _multipliers(real):
    """Q31 significand and power-of-two shift of each real multiplier, as an op's Prepare computes them."""
    frac, shift = np.frexp(np.asarray(real, np.float64))
    q = np.rint(frac * (1 << 31)).astype(np.int64)
    shift = shift.astype(np.int64)
    bump = q == (1 << 31)
    q[bump] //= 2
    shift[bump] += 1
    return torch.from_numpy(q.astype(np.int32)).cuda(), torch.from_numpy(shift.astype(np.int32)).cuda()


class _Model:
    """A decoder that gives its memory back when the program drops it."""

    def __init__(self, decoder):
        self.decoder = decoder

    def __del__(self):
        self.decoder.close()


def _decoder(g, seed, max_seq, max_batch, kv):
    """The Gemma-2B-shaped decoder with seeded random weights. The projections' scales are those of a real
    network rather than of a stress test: weights of standard deviation near 1 / sqrt(width), and the two
    that write to the residual stream smaller by sqrt(2 layers) as initialisation makes them, so that the
    attention's logits are of the order of one and the stream keeps its size over the layers."""
    weights = dec.make_weights(dec.GEMMA_2B, seed=seed)
    residual = 0.1 / math.sqrt(2 * dec.GEMMA_2B["n_layers"])
    for layer in weights["layers"]:
        for name in ("sq", "sk", "sv", "sgate", "sup"):
            layer[name].mul_(0.1)
        for name in ("so", "sdown"):
            layer[name].mul_(residual)
    weights["embed_scales"].mul_(2 / 3).add_(1e-2 / 3)  # rows of similar length, as a trained table has
    return _Model(dec.Decoder(dec.GEMMA_2B, max_seq=max_seq, max_batch=max_batch, weights=weights, kv_dtype=kv))


def _tokens(g, n):
    return torch.randint(0, dec.GEMMA_2B["vocab"], (n,), generator=g, device="cuda").to(torch.int32).cpu().numpy()


def prepare(case, seed):
    g = _rng(seed)
    c = dict(case)
    st = {"op": c["op"]}
    if c["op"] == "int8":
        m, n, k = c["m"], c["n"], c["k"]
        st["x"] = torch.randint(-128, 128, (m, k), generator=g, device="cuda").to(torch.int8)
        st["w"] = ops.PackedInt8Weights(_int8_weights(g, n, k))
        st["bias"] = torch.randint(-5000, 5001, (n,), generator=g, device="cuda").to(torch.int32)
        # the output scale covers the accumulators' spread: x of +-128 by weights of sigma 40
        w_scale = _uniform(g, 1e-3, 1e-2, n if c["per_channel"] else 1).cpu().numpy()
        out_scale = 0.02 * 5.5e-3 * 74.0 * math.sqrt(k)
        st["multipliers"], st["shifts"] = _multipliers(0.02 * w_scale.astype(np.float64) / out_scale)
        st["ws"] = ops.Workspace("cuda")
    elif c["op"] == "hybrid":
        m, n, k = c["m"], c["n"], c["k"]
        st["x"] = _normal(g, m, k)
        st["w"] = ops.PackedInt8Weights(_int8_weights(g, n, k))
        st["scales"] = _uniform(g, 1e-3, 1e-2, n)
        st["bias"] = _normal(g, n) if c["bias"] else None
        st["activation"], st["asymmetric"] = c["activation"], c["asymmetric"]
        st["ws"] = ops.Workspace("cuda")
    elif c["op"] == "int4":
        m, n, k = c["m"], c["n"], c["k"]
        st["x"] = _normal(g, m, k)
        nibbles = torch.randint(0, 256, (n, (k + 1) // 2), generator=g, device="cuda").to(torch.uint8)
        st["w"] = ops.PackedInt4Weights(nibbles, _uniform(g, 1e-3, 2e-2, n, k // c["block"]).half(), c["block"])
        st["ws"] = ops.Workspace("cuda")
    elif c["op"] == "sdpa":
        b, n, nkv, h, s = c["b"], c["n"], c["nkv"], c["h"], c["s_max"]
        lengths = torch.randint(max(1, s // 64), s + 1, (b,), generator=g, device="cuda").to(torch.int32)
        q, k, v = _normal(g, b, 1, n, h), _normal(g, b, s, nkv, h), _normal(g, b, s, nkv, h)
        st["args"] = dict(scale=1.0 / math.sqrt(h), logit_cap=c["cap"])
        if c["kv"] == "f32":
            # a graph's decode step: the cache's unwritten slots are masked out, no lengths
            past = torch.arange(s, device="cuda")[None, :] >= lengths[:, None]
            st["args"]["mask"] = torch.where(past, -1e30, 0.0).float()[:, None, None, :].contiguous()
        else:
            st["args"]["lengths"] = lengths
            q = q.half()
            if c["kv"] == "i8":
                for name, t in (("k_scale", k), ("v_scale", v)):
                    st["args"][name] = t.abs().amax(dim=-1).div_(127.0)
                    t.div_(st["args"][name][..., None]).round_().clamp_(-127, 127)
            dtype = torch.int8 if c["kv"] == "i8" else torch.float16
            k, v = k.to(dtype), v.to(dtype)
        st["q"], st["k"], st["v"] = q, k, v
        st["ws"] = ops.Workspace("cuda")
    elif c["op"] == "decode":
        b, ctx = c["batch"], c["context"]
        st["model"] = _decoder(g, seed, ctx + REPLY + 8, b, c["kv"])
        lengths = [ctx] * b
        if c["ragged"]:
            lengths = torch.randint((ctx + 1) // 2, ctx + 1, (b,), generator=g, device="cuda").cpu().tolist()
        d = st["model"].decoder
        for i, length in enumerate(lengths):
            d.prefill(_tokens(g, length), seq=i)
        st["positions"] = np.asarray(lengths, np.int32)
        st["tokens"] = _tokens(g, b)
    else:
        st["model"] = _decoder(g, seed, c["tokens"] + 8, 1, c["kv"])
        st["prompt"] = _tokens(g, c["tokens"])
        st["next"] = _tokens(g, 1)
    return st


# ---- one pass ------------------------------------------------------------------------------------------


def run(st):
    op = st["op"]
    if op == "int8":
        return ops.fully_connected_int8(st["x"], st["w"], st["bias"], -3, 0, st["multipliers"], st["shifts"], ws=st["ws"])
    if op == "hybrid":
        return ops.fully_connected_hybrid(st["x"], st["w"], st["scales"], st["bias"],
                                          asymmetric_quantize_inputs=st["asymmetric"], activation=st["activation"],
                                          ws=st["ws"])
    if op == "int4":
        return ops.fully_connected_blockwise4(st["x"], st["w"], ws=st["ws"])
    if op == "sdpa":
        return ops.sdpa_decode(st["q"], st["k"], st["v"], ws=st["ws"], **st["args"])
    d = st["model"].decoder
    if op == "decode":
        # a reply of REPLY tokens: the device feeds its own picks, the last step's logits come back too
        d.set_positions(st["positions"])
        tokens = d.run(st["tokens"], REPLY - 1)
        tokens, logits = d.step(tokens, want_logits=True)
        return tokens, logits
    # a prompt, and the probabilities behind the token that the program puts after it
    d.reset()
    first = d.prefill(st["prompt"])
    _, logits = d.step(st["next"], want_logits=True)
    return first, logits


# ---- floors and bounds ---------------------------------------------------------------------------------


def _projections():
    """int8 weights of one layer of the decoder."""
    c = dec.GEMMA_2B
    d, qd, kd = c["d_model"], c["n_heads"] * c["head_dim"], c["n_kv_heads"] * c["head_dim"]
    return d * (qd + 2 * kd) + qd * d + 3 * d * c["d_ff"]


def work(case):
    c = dict(case)
    if c["op"] in ("int8", "hybrid", "int4"):
        m, n, k = c["m"], c["n"], c["k"]
        flops = 2 * m * n * k
        if c["op"] == "int8":
            return {"bytes": m * k + n * k + 4 * n + (8 * n if c["per_channel"] else 8) + m * n, "flops": flops}
        if c["op"] == "hybrid":
            return {"bytes": 4 * m * k + n * k + 8 * n + (4 * n if c["bias"] else 0) + 4 * m * n, "flops": flops}
        return {"bytes": 4 * m * k + n * k // 2 + 2 * n * (k // c["block"]) + 4 * m * n, "flops": flops}
    if c["op"] == "sdpa":
        # lengths are uniform over the cache: half of it is read on average
        elem = {"f16": 2, "i8": 1, "f32": 4}[c["kv"]]
        tokens = c["b"] * (c["s_max"] + max(1, c["s_max"] // 64)) // 2
        rows = tokens * c["nkv"] * 2 * (c["h"] * elem + (4 if c["kv"] == "i8" else 0))
        qo = 2 * c["b"] * c["n"] * c["h"] * (4 if c["kv"] == "f32" else 2)
        return {"bytes": rows + qo + (4 * c["b"] * c["s_max"] if c["kv"] == "f32" else 4 * c["b"]),
                "flops": 4 * tokens * c["n"] * c["h"]}
    m = dec.GEMMA_2B
    head = m["vocab"] * m["d_model"]
    weights = m["n_layers"] * _projections()
    kv_row = 2 * m["n_layers"] * m["n_kv_heads"] * (m["head_dim"] * (1 if c["kv"] == "i8" else 2) + (4 if c["kv"] == "i8" else 0))
    attn = 4 * m["n_layers"] * m["n_heads"] * m["head_dim"]  # operations per query token and cached token
    if c["op"] == "decode":
        # the weights are far larger than what stays on the chip: every step of the reply reads them
        b, ctx = c["batch"], c["context"] * (0.75 if c["ragged"] else 1.0)
        return {"bytes": REPLY * (weights + head + b * ctx * kv_row) + 4 * b * m["vocab"],
                "flops": REPLY * b * (2 * (weights + head) + ctx * attn)}
    t = c["tokens"]
    # the prompt pass and the step behind it read the weights once each; the head sees two rows
    return {"bytes": 2 * (weights + head) + 2 * t * kv_row + 4 * m["vocab"],
            "flops": 2 * (t + 1) * weights + 4 * head + (t * (t + 1) // 2 + t) * attn}


def tolerance(case):
    if case["op"] == "int8":
        return "exact"
    if case["op"] == "hybrid":
        return {"rel": 1e-5}  # exact int32 sums, float32 scaling
    if case["op"] == "int4":
        # up to 8 rows: exact block sums added in float32; above: weight times block scale rounded to fp16
        return {"rel": 1e-5} if case["m"] <= 8 else {"rel": 1e-3}
    if case["op"] == "sdpa":
        return {"rel": 2e-3}  # fp16 operands and, but for float32 tensors, fp16 outputs
    # A last-bit difference in a sum moves an activation across an int8 rounding boundary somewhere in the 18
    # layers (each rounds to about 1/250 of the row's range) and the rest of the network carries it on.
    return {"rel": 2e-2, "max": 0.2, "differ": 0.01}
