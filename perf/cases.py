"""What this package is used for, as cases that can be timed: the transformer stacks of the Mimi codec on whole clips
and on live streams, the attention calls by themselves, and the two ends of the quantiser.

A case is a dict of plain values.  ``kind`` selects the path:

``clips``       eight transformer layers over whole clips (what an encoder or decoder transformer runs offline)
``stream``      the same eight layers for one call of ``frames`` new frames per live stream, on a KV ring
``attention``   projection + RoPE + banded attention of one layer, weights already in 16 bit
``window``      banded attention on given, rotated q, k, v in the layout the codec's attention modules hold them in
``quantise``    the encoder's end: stride-2 convolution, split residual vector quantiser -> codes
``dequantise``  the decoder's start: codes -> ordered sum and output projections -> transposed convolution

Sizes are frames of 40 ms (25 per second); the quantiser works on pairs of them.
"""
import math
import types

import torch

import fast_mimi_b200 as fm

LAYERS, HIDDEN, HEADS, HEAD_DIM, FFN, WINDOW = 8, 512, 8, 64, 2048, 250
ENTRIES, CODE_DIM = 2048, 256
STEPS = 16          # a stream's session covers this many calls, then starts again at the same position
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def listed():
    return [
        # a single 5 s utterance, as the codec's own examples encode it: FP32 model, one clip at a time
        {"name": "clips_one_5s", "kind": "clips", "batch": 1, "frames": 125, "dtype": "float32"},
        # offline encoding of a corpus in batches of 10 s clips with a BF16 model (one GPU's share of 512 clips on 8)
        {"name": "clips_64_10s", "kind": "clips", "batch": 64, "frames": 250, "dtype": "bfloat16"},
        # a few longer recordings of odd length, FP32 model
        {"name": "clips_6_24s", "kind": "clips", "batch": 6, "frames": 613, "dtype": "float32"},
        # one layer's attention over a full batch of 10 s clips, the benchmark's step
        {"name": "attention_512_10s", "kind": "attention", "batch": 512, "frames": 250, "dtype": "bfloat16"},
        # banded attention over 100 s recordings, called with a model's own FP32 q, k, v
        {"name": "window_16_100s", "kind": "window", "batch": 16, "frames": 2500, "dtype": "float32"},
        # one live conversation, one frame per call: the latency a listener hears
        {"name": "stream_1_frame", "kind": "stream", "streams": 1, "frames": 1, "past": 1000, "dtype": "float32"},
        # a server that advances a thousand live streams by one frame, rings full
        {"name": "stream_1024_frame", "kind": "stream", "streams": 1024, "frames": 1, "past": 5000, "dtype": "bfloat16"},
        # live streams fed at the codec's own rate of 12.5 codes per second: two frames per call
        {"name": "stream_64_pairs", "kind": "stream", "streams": 64, "frames": 2, "past": 375, "dtype": "float32"},
        # a handful of recordings encoded in 2 s chunks as they arrive
        {"name": "stream_5_chunks", "kind": "stream", "streams": 5, "frames": 50, "past": 130, "dtype": "float32"},
        # codes of the single 5 s utterance
        {"name": "quantise_one_5s", "kind": "quantise", "batch": 1, "frames": 125, "quantizers": 8},
        # codes of the full batch of 10 s clips
        {"name": "quantise_512_10s", "kind": "quantise", "batch": 512, "frames": 250, "quantizers": 8},
        # decoding a batch of 10 s clips: what the decoder transformer is handed
        {"name": "dequantise_64_10s", "kind": "dequantise", "batch": 64, "frames": 250, "quantizers": 8},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["clips", "clips", "stream", "stream", "attention", "window", "quantise", "dequantise"])
    if kind == "clips":
        frames = _log(rng, 17, 2500)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 16000 // frames)), "frames": frames,
                "dtype": rng.choice(["float32", "float32", "bfloat16", "float16"])}
    if kind == "stream":
        frames = rng.choice([1, 1, 1, 2, 2, _log(rng, 3, 150)])
        return {"kind": kind, "streams": _log(rng, 1, max(1, min(1024, 4000 // frames))), "frames": frames,
                "past": _log(rng, 1, 3000) - 1, "dtype": rng.choice(["float32", "float32", "bfloat16"])}
    if kind == "attention":
        frames = _log(rng, 33, 2500)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 128000 // frames)), "frames": frames,
                "dtype": rng.choice(["bfloat16", "float16"])}
    if kind == "window":
        frames = _log(rng, 33, 2500)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 40000 // frames)), "frames": frames,
                "dtype": rng.choice(["float32", "bfloat16", "float16"])}
    frames = _log(rng, 25, 1500)
    quantizers = rng.choice([8, 8, 16, 32])
    most = 128000 * 8 // quantizers if kind == "quantise" else 64000
    return {"kind": kind, "batch": _log(rng, 1, max(1, most // frames)), "frames": frames, "quantizers": quantizers}


# ------------------------------------------------------------------------------------------------- what a program holds
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, *shape, std=1.0, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=gen)


def _layers(gen, dtype):
    """A stack as a program holds it: matrices ~ N(0, 1 / fan_in), LayerNorm weights around one, layer scales of 0.1
    (ten times the initial value, so that every branch shows in the stack's output)."""
    with torch.device("cuda"):
        layers = [fm.MimiTransformerLayerB200(layer_idx=i) for i in range(LAYERS)]
    with torch.no_grad():
        for layer in layers:
            for name, p in layer.named_parameters():
                p.requires_grad_(False)
                if name.endswith("scale.scale"):
                    p.fill_(0.1)
                elif name.endswith("layernorm.weight"):
                    p.uniform_(0.9, 1.1, generator=gen)
                elif name.endswith("layernorm.bias"):
                    p.normal_(0.0, 0.01, generator=gen)
                else:
                    p.normal_(0.0, p.shape[1] ** -0.5, generator=gen)
    return [layer.to(dtype).eval() for layer in layers]


def _quantiser(gen, quantizers):
    """One semantic stack and the acoustic stacks behind it; codebooks get finer with depth, as trained ones do."""
    def branch(n):
        scale = 0.6 ** torch.arange(n, device="cuda", dtype=torch.float32).clamp(max=7)
        books = _normal(gen, n, ENTRIES, CODE_DIM) * scale[:, None, None]
        return fm.MimiRVQB200(books, _normal(gen, CODE_DIM, HIDDEN, 1, std=HIDDEN ** -0.5),
                              _normal(gen, HIDDEN, CODE_DIM, 1, std=CODE_DIM ** -0.5))
    return fm.MimiSplitRVQB200(branch(1), branch(quantizers - 1))


def prepare(case, seed):
    gen = _generator(seed)
    kind, frames = case["kind"], case["frames"]
    state = {"kind": kind}
    if kind == "clips":
        dtype = DTYPES[case["dtype"]]
        state["layers"] = _layers(gen, dtype)
        state["x"] = _normal(gen, case["batch"], frames, HIDDEN, dtype=dtype)
        state["positions"] = fm.rope_tables(torch.arange(frames, device="cuda")[None])
    elif kind == "stream":
        dtype, streams, past = DTYPES[case["dtype"]], case["streams"], case["past"]
        state["layers"] = _layers(gen, dtype)
        state["x"] = _normal(gen, streams, frames, HIDDEN, dtype=dtype)
        state["cos"], state["sin"] = fm.rope_tables(torch.arange(past, past + STEPS * frames, device="cuda")[None])
        state["cache"] = fm.MimiKVRing(LAYERS, streams, WINDOW, device="cuda")
        state["cache"].ring_k.normal_(0.0, 1.0, generator=gen)
        state["cache"].ring_v.normal_(0.0, 1.0, generator=gen)
        state.update(past=past, frames=frames, turn=STEPS)
    elif kind == "attention":
        dtype = DTYPES[case["dtype"]]
        state["x"] = _normal(gen, case["batch"], frames, HIDDEN, dtype=dtype)
        state["w"] = _normal(gen, 3 * HIDDEN, HIDDEN, std=0.02, dtype=dtype)
        state["positions"] = fm.rope_tables(torch.arange(frames, device="cuda")[None])
    elif kind == "window":
        # [B, T, 8, 64] seen as [B, 8, T, 64]: how projections leave q, k, v
        state["qkv"] = [_normal(gen, case["batch"], frames, HEADS, HEAD_DIM, std=0.125, dtype=DTYPES[case["dtype"]])
                        .transpose(1, 2) for _ in range(3)]
    elif kind == "quantise":
        conv = torch.nn.Conv1d(HIDDEN, HIDDEN, 4, 2, bias=False, device="cuda").requires_grad_(False)
        conv.weight.normal_(0.0, (4 * HIDDEN) ** -0.5, generator=gen)
        state["down"] = fm.MimiDownsampleB200(types.SimpleNamespace(conv=conv, causal=True, pad_mode="replicate"))
        state["quantiser"], state["quantizers"] = _quantiser(gen, case["quantizers"]), case["quantizers"]
        state["x"] = _normal(gen, case["batch"], frames, HIDDEN, std=1.5)
    else:
        conv = torch.nn.ConvTranspose1d(HIDDEN, HIDDEN, 4, 2, groups=HIDDEN, bias=False, device="cuda").requires_grad_(False)
        conv.weight.normal_(0.0, 0.5, generator=gen)
        state["up"] = fm.MimiUpsampleB200(types.SimpleNamespace(conv=conv, padding_left=0, padding_right=2))
        state["quantiser"] = _quantiser(gen, case["quantizers"])
        state["codes"] = torch.randint(0, ENTRIES, (case["batch"], case["quantizers"], (frames + 1) // 2), device="cuda",
                                       generator=gen)
    return state


# ------------------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    with torch.no_grad():
        if kind == "clips":
            h = state["x"]
            for layer in state["layers"]:
                h, _ = layer(h, None, None, state["positions"])
            return h
        if kind == "stream":
            cache, n = state["cache"], state["frames"]
            if state["turn"] == STEPS:                  # a new session at the same position, over the same rings
                state["turn"] = 0
                cache.reset()
                for i in range(LAYERS):
                    cache.advance(i, state["past"])
            at = state["turn"] * n
            state["turn"] += 1
            positions = state["cos"][:, at:at + n], state["sin"][:, at:at + n]
            h = state["x"]
            for layer in state["layers"]:
                h, _ = layer(h, None, cache, positions)
            return {"hidden": h, "ring_k": cache.ring_k, "ring_v": cache.ring_v}
        if kind == "attention":
            return fm.ops.attention_prefill(state["x"], state["w"], *state["positions"], window=WINDOW)
        if kind == "window":
            return fm.native_window_attention(*state["qkv"], scale=HEAD_DIM ** -0.5, window=WINDOW)
        if kind == "quantise":
            embeddings = state["down"](state["x"].transpose(1, 2))
            return {"embeddings": embeddings, "codes": state["quantiser"].encode(embeddings, state["quantizers"])}
        embeddings = state["up"](state["quantiser"].decode(state["codes"]))
        return embeddings.transpose(1, 2)


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(queries, past=0):
    """(query, key) pairs of one clip or stream under the window."""
    return sum(min(past + i + 1, WINDOW) for i in range(queries))


def work(case):
    kind, frames = case["kind"], case["frames"]
    size = 4 if case.get("dtype", "float32") == "float32" else 2
    layer_weights = HIDDEN * (3 * HIDDEN + HIDDEN + 2 * FFN)
    if kind == "clips":
        rows = case["batch"] * frames
        return {"bytes": LAYERS * layer_weights * 2 + 2 * rows * HIDDEN * size + 2 * frames * HEAD_DIM * 4,
                "flops": LAYERS * (2 * layer_weights * rows + 4 * HIDDEN * case["batch"] * _pairs(frames))}
    if kind == "stream":
        streams = case["streams"]
        rows, past = streams * frames, case["past"]
        ring = 2 * 2 * HIDDEN * (streams * min(past, WINDOW - 1) + rows)       # K and V rows read, new rows written
        return {"bytes": LAYERS * (layer_weights * 2 + ring) + 2 * rows * HIDDEN * size,
                "flops": LAYERS * (2 * layer_weights * rows + 4 * HIDDEN * streams * _pairs(frames, past))}
    if kind == "attention":
        rows = case["batch"] * frames
        return {"bytes": 2 * rows * HIDDEN * 2 + 3 * HIDDEN * HIDDEN * 2 + 2 * frames * HEAD_DIM * 4,
                "flops": 2 * 3 * HIDDEN * HIDDEN * rows + 4 * HIDDEN * case["batch"] * _pairs(frames)}
    if kind == "window":
        return {"bytes": 4 * case["batch"] * frames * HIDDEN * size, "flops": 4 * HIDDEN * case["batch"] * _pairs(frames)}
    rows, n = case["batch"] * ((frames + 1) // 2), case["quantizers"]
    if kind == "quantise":
        weights = 4 * HIDDEN * HIDDEN + 2 * CODE_DIM * HIDDEN + n * ENTRIES * CODE_DIM
        return {"bytes": 4 * (weights + case["batch"] * frames * HIDDEN + rows * HIDDEN) + 8 * rows * n,
                "flops": 2 * rows * weights}
    return {"bytes": 8 * rows * n + 4 * (n * min(rows, ENTRIES) * CODE_DIM + 2 * CODE_DIM * HIDDEN + 2 * rows * HIDDEN),
            "flops": rows * (n * CODE_DIM + 2 * 2 * CODE_DIM * HIDDEN + 2 * 4 * HIDDEN)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("clips", "stream"):
        # FP32 residual streams: 16-bit operands of the products (2^-11 each) seen through layer scales of 0.1.
        # 16-bit residual streams are rounded sixteen times on the way (2^-9 for BF16, 2^-11 for FP16).
        return {"rel": {"float32": 1e-3, "float16": 3e-3, "bfloat16": 1e-2}[case["dtype"]]}
    if kind in ("attention", "window"):
        return {"rel": 3e-3}              # q, k in BF16, probabilities, v and result in 16 bit
    if kind == "quantise":
        # FP32-grade embeddings; where two entries are equally near to the last FP32 bits either is right, and the
        # residual layers behind such a choice differ with it
        return {"rel": 1e-5, "differ": 2e-3}
    return {"rel": 1e-5}
