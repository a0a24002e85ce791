"""What is timed: the work a program that serves quantized models has this package do.

Every case goes through the public surface (the modules of ``mlx_kquant_b200.nn``, the ops, the mixture-of-experts
block). ``listed()`` is the fixed set, ``draw(rng)`` gives further cases of the same ranges:

  linear   one eager ``KQuantLinear`` call: a single row (latency of a call), a batch of decode rows, a prefill
  chain    a decode step over square layers, each consuming the output of the one before, replayed as a CUDA graph
  layer    the projections of decoder layers (output projection, SwiGLU feed-forward, residuals and norms between
           them) for a few rows, replayed as a CUDA graph: what one decode step of a dense model calls
  mlp      the feed-forward of one layer over a prompt, eager
  dequant  wire bytes to floats: an embedding or output matrix expanded once
  heads    the per-head projections of absorbed attention, both orientations, one decode step
  moe      router, 128-expert SwiGLU block, weighted sum: decode batches as CUDA graphs, prompts eager

A decode step is replayed from a graph because that is how launch-bound steps are served; the graph and its static
input are what such a program keeps. A pass is the steps of two consecutive tokens with activations of their own:
each step's input is copied in, the graph replayed, the step's result copied out - so every intermediate buffer
holds the values of another token when a step begins, as it does in a decode loop. Weights are codec blocks that the
host encoder made from normally distributed rows with the variance of trained matrices (1 / inputs, so that a chain of
products keeps its magnitude), drawn with replacement from a pool of encoded blocks; activations are N(0, 1). ``kq.quantize`` is not timed: it converts checkpoints on the host,
offline.
"""
from __future__ import annotations

import math

import torch

import mlx_kquant_b200 as kq
from mlx_kquant_b200 import moe
from mlx_kquant_b200.nn import KQuantLinear, KQuantMultiLinear

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
SUPER = ("q4_k", "q6_k", "q5_k", "q3_k", "q2_k", "iq4_xs", "iq2_xxs")   # 256 weights per block
SMALL = ("q8_0", "q4_0", "iq4_nl", "q4_1", "q5_0", "q5_1")              # 32 weights per block
#: multiply-adds of the largest drawn product: those of the largest listed case
MOST_MACS = 8192 * 14336 * 4096
#: decode steps of one pass of a case that is replayed from a graph
TOKENS = 2


def listed():
    return [
        # the smallest call: one token through one projection, no graph - what an interactive program pays per call
        {"name": "call_q4k_1row", "kind": "linear", "codec": "q4_k", "m": 1, "n": 4096, "k": 4096, "dtype": "bf16"},
        # one token through 32 square projections, each waiting for the one before (the benchmark's matrix)
        {"name": "token_q4k_chain", "kind": "chain", "codec": "q4_k", "m": 1, "k": 4096, "layers": 32, "dtype": "f16"},
        # one token through two decoder layers of a Llama-3-8B-class model in the usual q4_k / q6_k mix
        {"name": "token_mixed_layers", "kind": "layer", "codec": "q4_k", "codec_down": "q6_k", "m": 1, "hidden": 4096,
         "ffn": 14336, "layers": 2, "dtype": "bf16"},
        # eight concurrent sequences (or a speculative window) through the same layers
        {"name": "batch8_mixed_layers", "kind": "layer", "codec": "q4_k", "codec_down": "q6_k", "m": 8, "hidden": 4096,
         "ffn": 14336, "layers": 2, "dtype": "bf16"},
        # four rows through a 70B-class projection in a 4-bit IQ codec
        {"name": "iq4xs_4rows", "kind": "linear", "codec": "iq4_xs", "m": 4, "n": 28672, "k": 8192, "dtype": "f16"},
        # a serving batch of 61 sequences through a 70B-class projection: many rows, still bound by the weights
        {"name": "batch61_q4k", "kind": "linear", "codec": "q4_k", "m": 61, "n": 28672, "k": 8192, "dtype": "bf16"},
        # a prompt of 509 tokens through a feed-forward: a ragged number of rows, three products
        {"name": "prefill509_mlp", "kind": "mlp", "codec": "q4_k", "codec_down": "q6_k", "m": 509, "hidden": 4096,
         "ffn": 14336, "dtype": "bf16"},
        # the largest: a batch of long prompts through one projection
        {"name": "prefill8192_q4k", "kind": "linear", "codec": "q4_k", "m": 8192, "n": 14336, "k": 4096,
         "dtype": "bf16"},
        # an output matrix expanded to floats
        {"name": "dequant_q6k", "kind": "dequant", "codec": "q6_k", "n": 14336, "k": 4096, "dtype": "bf16"},
        # absorbed attention, eight sequences, eight layers: query up-projection (transpose=False), value projection
        {"name": "heads_absorbed", "kind": "heads", "codec": "q6_k", "heads": 64, "head_dim": 128, "rank": 512,
         "batch": 8, "layers": 8, "dtype": "bf16"},
        # mixture of experts, a decode batch: every expert has a handful of rows
        {"name": "moe_batch64", "kind": "moe", "codec": "q4_k", "tokens": 64, "experts": 128, "top_k": 8,
         "hidden": 2048, "ffn": 768, "graph": True, "dtype": "bf16"},
        # mixture of experts over a prompt
        {"name": "moe_prompt4096", "kind": "moe", "codec": "q4_k", "tokens": 4096, "experts": 128, "top_k": 8,
         "hidden": 2048, "ffn": 768, "graph": False, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer of [lo, hi], a multiple of `step`, spread evenly over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "chain", "layer", "layer", "mlp", "dequant", "heads", "moe", "moe"))
    act = rng.choice(("bf16", "bf16", "f16"))
    main = rng.choice(("q4_k", "q4_k", "q4_k", "q6_k", "q6_k", "q5_k", "q3_k", "q8_0", "iq4_xs", "q4_0"))
    if kind == "linear":
        codec = rng.choice(("q4_k", "q4_k", "q6_k") + SUPER + SMALL)
        step = 256 if codec in SUPER else 32
        n, k = _log_int(rng, 256, 28672), _log_int(rng, 512, 14336, step)
        m = _log_int(rng, 1, 8192)
        m = max(1, min(m, MOST_MACS // (n * k)))
        return {"kind": kind, "codec": codec, "m": m, "n": n, "k": k,
                "dtype": rng.choice(("bf16", "bf16", "f16", "f32"))}
    if kind == "chain":
        k = _log_int(rng, 1024, 8192, 256)
        return {"kind": kind, "codec": main, "m": _log_int(rng, 1, 16), "k": k,
                "layers": max(2, min(32, (32 * 4096 * 4096) // (k * k))), "dtype": act}
    if kind == "layer":
        return {"kind": kind, "codec": main, "codec_down": rng.choice(("q6_k", "q6_k", main)),
                "m": _log_int(rng, 1, 64), "hidden": _log_int(rng, 1024, 8192, 256),
                "ffn": _log_int(rng, 2048, 14336, 256), "layers": rng.randint(1, 3), "dtype": act}
    if kind == "mlp":
        return {"kind": kind, "codec": main, "codec_down": rng.choice(("q6_k", "q6_k", main)),
                "m": _log_int(rng, 17, 2048), "hidden": _log_int(rng, 1024, 4096, 256),
                "ffn": _log_int(rng, 2048, 14336, 256), "dtype": act}
    if kind == "dequant":
        codec = rng.choice(SUPER + SMALL)
        return {"kind": kind, "codec": codec, "n": _log_int(rng, 64, 14336),
                "k": _log_int(rng, 512, 8192, 256 if codec in SUPER else 32),
                "dtype": rng.choice(("f16", "bf16", "f32"))}
    if kind == "heads":
        return {"kind": kind, "codec": rng.choice(("q4_k", "q6_k", "q8_0")), "heads": rng.choice((16, 32, 64, 128)),
                "head_dim": rng.choice((64, 128, 192)), "rank": rng.choice((256, 512)), "batch": _log_int(rng, 1, 16),
                "layers": rng.randint(2, 8), "dtype": act}
    tokens = _log_int(rng, 1, 4096)
    experts = rng.choice((16, 60, 64, 128))
    return {"kind": "moe", "codec": rng.choice(("q4_k", "q4_k", "q4_k", "q6_k")), "tokens": tokens, "experts": experts,
            "top_k": rng.choice((2, 4, 8)), "hidden": 256 * rng.randint(4, 8), "ffn": 256 * rng.randint(2, 3),
            "graph": tokens <= 512, "dtype": act}


def _wire(codec, n, k, gen, lead=(), std=None):
    """uint8 lead + [n, bytes of k weights]: blocks encoded from N(0, std), by default 1 / sqrt(k), drawn from a pool."""
    wpb, bpb, _, needs_imatrix = kq.codec_geometry(codec)
    pool_blocks = 128 if codec == "iq2_xxs" else 512
    rows = torch.randn((pool_blocks, wpb), generator=gen, device="cuda").mul_(std or k ** -0.5).cpu()
    pool, _ = kq.quantize(rows, codec, torch.ones(wpb) if needs_imatrix else None)
    pick = torch.randint(0, pool_blocks, tuple(lead) + (n, k // wpb), generator=gen, device="cuda", dtype=torch.int32)
    return pool.cuda()[pick].reshape(tuple(lead) + (n, k // wpb * bpb))


class _Package:
    """The path's steps as this package offers them."""

    @staticmethod
    def linear(codec, w, k):
        with torch.device("cuda"):
            layer = KQuantLinear(k, w.shape[0], False, codec)
        layer.weight = w
        return layer

    @staticmethod
    def heads(codec, w, k):
        with torch.device("cuda"):
            layer = KQuantMultiLinear(k, w.shape[1], w.shape[0], codec)
        layer.weight = w
        return layer

    norm = staticmethod(lambda x: torch.nn.functional.rms_norm(x, (x.shape[-1],)))
    swiglu = staticmethod(moe.swiglu)
    dequantize = staticmethod(kq.dequantize)

    @staticmethod
    def block(x, logits, top_k, gate, up, down, codec):
        gate_up = moe.fuse_gate_up(gate, up)

        def block(x, logits):
            ids, probs = moe.route_topk(logits, top_k)
            return moe.moe_glu(x, None, None, down, codec, ids, probs, w_gate_up=gate_up)
        return [x, logits], block


class _Double:
    """The same steps in plain torch and float64, no value rounded between them."""

    @staticmethod
    def linear(codec, w, k):
        return lambda x: x.double() @ _decode(codec, w).T

    @staticmethod
    def heads(codec, w, k):
        def product(x, transpose=True):
            d = _decode(codec, w)
            return torch.einsum("bhlk,hnk->bhln" if transpose else "bhln,hnk->bhlk", x.double(), d)
        return product

    @staticmethod
    def norm(x):
        eps = torch.finfo(torch.float32).eps   # what rms_norm takes for rows of 16-bit and 32-bit floats
        return x * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + eps)

    swiglu = staticmethod(lambda gate, up: torch.nn.functional.silu(gate) * up)
    dequantize = staticmethod(lambda w, scales, codec, dtype: _decode(codec, w))

    @staticmethod
    def block(x, logits, top_k, gate, up, down, codec):
        def block(x, logits):
            x, scores = x.double(), torch.softmax(logits.double(), -1)
            scores, ids = scores.topk(top_k, dim=-1)
            scores = scores / scores.sum(-1, keepdim=True)
            y = torch.zeros_like(x)
            for e in range(gate.shape[0]):
                t, slot = (ids == e).nonzero(as_tuple=True)
                h = _Double.swiglu(x[t] @ _decode(codec, gate[e]).T, x[t] @ _decode(codec, up[e]).T)
                y.index_add_(0, t, h @ _decode(codec, down[e]).T * scores[t, slot, None])
            return y
        return [x, logits], block


def _randn(shape, dtype, gen):
    return torch.randn(shape, generator=gen, device="cuda").to(DTYPES[dtype])


def _step_fn(case, gen, lib):
    """(inputs, fn): fn(*inputs) is one pass; lib: whose steps it is made of."""
    kind, codec, dtype = case["kind"], case["codec"], case["dtype"]

    def linear(codec, n, k):
        return lib.linear(codec, _wire(codec, n, k, gen), k)
    if kind == "linear":
        layer = linear(codec, case["n"], case["k"])
        return [_randn((case["m"], case["k"]), dtype, gen)], layer
    if kind == "chain":
        layers = [linear(codec, case["k"], case["k"]) for _ in range(case["layers"])]

        def chain(x):
            for layer in layers:
                x = layer(x)
            return x
        return [_randn((case["m"], case["k"]), dtype, gen)], chain
    if kind in ("layer", "mlp"):
        h, f, down = case["hidden"], case["ffn"], case["codec_down"]
        blocks = [(linear(codec, h, h) if kind == "layer" else None, linear(codec, f, h), linear(codec, f, h),
                   linear(down, h, f)) for _ in range(case.get("layers", 1))]

        def feed_forward(gate, up, down, x):
            return down(lib.swiglu(gate(x), up(x)))

        def mlp(x):
            return feed_forward(*blocks[0][1:], x)

        def decoder(x):
            for out_proj, *ffn in blocks:
                x = x + out_proj(lib.norm(x))
                x = x + feed_forward(*ffn, lib.norm(x))
            return x
        return [_randn((case["m"], h), dtype, gen)], decoder if kind == "layer" else mlp
    if kind == "dequant":
        w = _wire(codec, case["n"], case["k"], gen)
        return [w], lambda w: lib.dequantize(w, None, codec, DTYPES[dtype])
    if kind == "heads":
        nh, d, r, b = case["heads"], case["head_dim"], case["rank"], case["batch"]

        def heads():   # used in both orientations: d inputs one way, r the other
            return lib.heads(codec, _wire(codec, d, r, gen, lead=(nh,), std=(d * r) ** -0.25), r)
        layers = [(heads(), heads()) for _ in range(case["layers"])]

        def attention(q):
            for q_up, v_down in layers:   # the attention between the two is not this package's work
                q = v_down(q_up(q, transpose=False))
            return q
        return [_randn((b, nh, 1, d), dtype, gen)], attention
    h, f, e = case["hidden"], case["ffn"], case["experts"]
    gate, up = _wire(codec, f, h, gen, lead=(e,)), _wire(codec, f, h, gen, lead=(e,))
    down = _wire(codec, h, f, gen, lead=(e,))
    x, logits = _randn((case["tokens"], h), dtype, gen), torch.randn((case["tokens"], e), generator=gen, device="cuda")
    return lib.block(x, logits, case["top_k"], gate, up, down, codec)


def _inputs(case, seed, lib):
    """(the inputs of every step, fn): a case that is replayed from a graph has two steps, any other one."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    inputs, fn = _step_fn(case, gen, lib)
    if not (case["kind"] in ("chain", "layer", "heads") or case.get("graph")):
        return [inputs], fn
    return [inputs, [torch.randn(x.shape, generator=gen, device="cuda").to(x.dtype) for x in inputs]], fn


def prepare(case, seed):
    steps, fn = _inputs(case, seed, _Package)
    inputs = steps[0]
    if len(steps) == 1:
        return {"inputs": inputs, "fn": fn}
    static = [x.clone() for x in inputs]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            fn(*static)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        output = fn(*static)
    # fn holds the weights, which the graph reads
    return {"steps": steps, "static": static, "graph": graph, "output": output, "fn": fn,
            "results": [torch.empty_like(output) for _ in range(TOKENS)]}


def run(state):
    if "graph" not in state:
        return state["fn"](*state["inputs"])
    for inputs, result in zip(state["steps"], state["results"]):
        for dst, src in zip(state["static"], inputs):
            dst.copy_(src)
        state["graph"].replay()
        result.copy_(state["output"])
    return state["results"]


def _bytes(codec, weights):
    wpb, bpb, _, _ = kq.codec_geometry(codec)
    return weights // wpb * bpb


def work(case):
    """Wire bytes of the weights that are used, activations in and out once, two flops per multiply-add."""
    kind, codec = case["kind"], case["codec"]
    item = 4 if case["dtype"] == "f32" else 2
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _bytes(codec, n * k) + m * (k * item + n * 2), "flops": 2 * m * n * k}
    if kind == "chain":
        m, k, layers = case["m"], case["k"], case["layers"]
        return {"bytes": TOKENS * (layers * _bytes(codec, k * k) + 2 * m * k * item),
                "flops": TOKENS * 2 * m * k * k * layers}
    if kind in ("layer", "mlp"):
        m, h, f, layers = case["m"], case["hidden"], case["ffn"], case.get("layers", 1)
        first, steps = (h * h, TOKENS) if kind == "layer" else (0, 1)
        wire = _bytes(codec, first + 2 * h * f) + _bytes(case["codec_down"], h * f)
        return {"bytes": steps * (layers * wire + 2 * m * h * item), "flops": steps * 2 * m * layers * (first + 3 * h * f)}
    if kind == "dequant":
        weights = case["n"] * case["k"]
        return {"bytes": _bytes(codec, weights) + weights * item, "flops": 0}
    if kind == "heads":
        nh, d, r, b, layers = case["heads"], case["head_dim"], case["rank"], case["batch"], case["layers"]
        return {"bytes": TOKENS * 2 * (layers * _bytes(codec, nh * d * r) + b * nh * d * item),
                "flops": TOKENS * 4 * b * nh * d * r * layers}
    t, h, f, e, top_k = case["tokens"], case["hidden"], case["ffn"], case["experts"], case["top_k"]
    touched = e * (1.0 - (1.0 - top_k / e) ** t)   # experts that at least one token is expected to choose
    steps = TOKENS if case["graph"] else 1
    return {"bytes": steps * (touched * _bytes(codec, 3 * h * f) + t * (2 * h * item + e * 4)),
            "flops": steps * 6 * t * top_k * h * f}


def tolerance(case):
    """Dequantization is exact. Products: about four times the distance measured between this package and the same
    steps on weights expanded to float32 (sums in float32 or float64, every result rounded to the activation type
    where the package rounds it). One rounding of the output is most of it: 2^-9 (bf16) or 2^-12 (f16) of a value
    on average; chained steps and the products of a gated feed-forward add up such roundings."""
    kind = case["kind"]
    half = case["dtype"] == "f16"
    if kind == "dequant":
        return "exact"
    if kind == "linear":                                               # seen: 1.3e-3 / 8e-3, f16 3.3e-4 / 1.4e-3
        return {"rel": 1.2e-3, "max": 6e-3} if half else {"rel": 5e-3, "max": 3e-2}
    if kind == "chain":                                                # seen: 1.2e-2 / 6e-2, f16 2.6e-3 / 1.1e-2
        return {"rel": 1e-2, "max": 5e-2} if half else {"rel": 3e-2, "max": 0.2}
    if kind == "heads":                                                # seen: 5.1e-3 / 3.4e-2, f16 2.3e-3 / 5.3e-3
        return {"rel": 8e-3, "max": 2e-2} if half else {"rel": 2e-2, "max": 0.12}
    if kind == "layer":                                                # seen: 8.4e-3 / 3.5e-2, f16 1.2e-3 / 5.3e-3
        return {"rel": 5e-3, "max": 2.5e-2} if half else {"rel": 2.5e-2, "max": 0.12}
    if kind == "mlp":                                                  # seen: 3.0e-3 / 1.3e-2, f16 9.3e-4 / 4.7e-3
        return {"rel": 4e-3, "max": 2e-2} if half else {"rel": 1.2e-2, "max": 5e-2}
    return {"rel": 2.5e-3, "max": 1e-2} if half else {"rel": 1.5e-2, "max": 0.1}   # seen: 4.7e-3 / 2.5e-2, f16 6e-4


def _half(b, at):
    """The float16 at byte `at` of every block, as [blocks, 1] float64."""
    return b[:, at:at + 2].contiguous().view(torch.float16).double()


def _nibbles(q, run):
    """Bytes [blocks, n] -> [blocks, n / run, 2, run]: the low nibbles of every run of bytes, then its high ones."""
    q = q.reshape(q.shape[0], -1, 1, run)
    return torch.cat((q & 15, q >> 4), 2)


def _bits(q, at, count, width):
    """`count` fields of `width` bits from bit `at` upwards of every byte: [blocks, count, bytes]."""
    shift = torch.arange(at, at + count * width, width, device=q.device)
    return (q[:, None] >> shift[:, None]) & ((1 << width) - 1)


IQ4 = (-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113)


def _scales_mins(b):
    """q4_k / q5_k: the eight 6-bit scales and mins of a block's twelve packed bytes, [blocks, 8, 1] each."""
    lo, mid, hi = b[:, 0:4], b[:, 4:8], b[:, 8:12]
    sc = torch.cat((lo & 63, (hi & 15) | (lo >> 6 << 4)), 1)
    mn = torch.cat((mid & 63, (hi >> 4) | (mid >> 6 << 4)), 1)
    return sc[..., None].double(), mn[..., None].double()


def _decode(codec, wire):
    """Wire bytes -> float64 weights, from the block formats' definitions. iq2_xxs (a lattice of 256 points that no
    formula gives) has no decoder here: exact() says None for it."""
    wpb, bpb, _, _ = kq.codec_geometry(codec)
    b = wire.reshape(-1, bpb)
    n = b.shape[0]
    i = b.int()
    if codec == "q8_0":
        v = _half(b, 0) * b[:, 2:].contiguous().view(torch.int8).double()
    elif codec == "q4_0":
        v = _half(b, 0) * (_nibbles(i[:, 2:], 16).reshape(n, 32) - 8)
    elif codec == "q4_1":
        v = _half(b, 0) * _nibbles(i[:, 4:], 16).reshape(n, 32) + _half(b, 2)
    elif codec in ("q5_0", "q5_1"):
        at = 2 if codec == "q5_0" else 4
        high = _bits(i[:, at:at + 4], 0, 8, 1).transpose(1, 2).reshape(n, 32)
        q = _nibbles(i[:, at + 4:], 16).reshape(n, 32) | high << 4
        v = _half(b, 0) * (q - 16) if codec == "q5_0" else _half(b, 0) * q + _half(b, 2)
    elif codec in ("iq4_nl", "iq4_xs"):
        levels = torch.tensor(IQ4, device=b.device, dtype=torch.float64)
        v = levels[_nibbles(i[:, 2 if codec == "iq4_nl" else 8:], 16).long()].reshape(n, -1, 32)
        if codec == "iq4_xs":
            low = torch.stack((i[:, 4:8] & 15, i[:, 4:8] >> 4), 2).reshape(n, 8)
            high = _bits(i[:, 2:4], 0, 4, 2).transpose(1, 2).reshape(n, 8)
            v = v * ((low | high << 4) - 32)[..., None]
        v = v * _half(b, 0)[..., None]
    elif codec == "q4_k":
        sc, mn = _scales_mins(i[:, 4:16])
        v = _half(b, 0)[..., None] * sc * _nibbles(i[:, 16:], 32).reshape(n, 8, 32) - _half(b, 2)[..., None] * mn
    elif codec == "q5_k":
        sc, mn = _scales_mins(i[:, 4:16])
        q = _nibbles(i[:, 48:], 32).reshape(n, 8, 32) | _bits(i[:, 16:48], 0, 8, 1) << 4
        v = _half(b, 0)[..., None] * sc * q - _half(b, 2)[..., None] * mn
    elif codec == "q6_k":
        q = torch.cat([_nibbles(i[:, 64 * h:64 * h + 64], 64).reshape(n, 4, 32)
                       | _bits(i[:, 128 + 32 * h:160 + 32 * h], 0, 4, 2) << 4 for h in (0, 1)], 1) - 32
        sc = b[:, 192:208].contiguous().view(torch.int8).double()
        v = _half(b, 208)[..., None] * sc[..., None] * q.reshape(n, 16, 16)
    elif codec == "q3_k":
        q = torch.cat([_bits(i[:, 32 + 32 * h:64 + 32 * h], 0, 4, 2) for h in (0, 1)], 1)
        q = q + 4 * _bits(i[:, :32], 0, 8, 1) - 4
        sc = torch.cat((i[:, 96:104] & 15, i[:, 96:104] >> 4), 1) | _bits(i[:, 104:108], 0, 4, 2).reshape(n, 16) << 4
        v = _half(b, 108)[..., None] * (sc - 32)[..., None] * q.reshape(n, 16, 16)
    elif codec == "q2_k":
        q = torch.cat([_bits(i[:, 16 + 32 * h:48 + 32 * h], 0, 4, 2) for h in (0, 1)], 1).reshape(n, 16, 16)
        v = _half(b, 80)[..., None] * (i[:, :16] & 15)[..., None] * q - _half(b, 82)[..., None] * (i[:, :16] >> 4)[..., None]
    else:
        raise NotImplementedError(codec)
    return v.reshape(wire.shape[:-1] + (wire.shape[-1] // bpb * wpb,))


def exact(case, seed):
    if "iq2_xxs" in (case["codec"], case.get("codec_down")):
        return None
    steps, fn = _inputs(case, seed, _Double)
    outputs = [fn(*inputs) for inputs in steps]
    return outputs if len(steps) > 1 else outputs[0]
