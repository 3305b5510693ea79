"""The kernels that calls with few rows take: the split-K linear and projection (128 x 64 tiles, K shared out over a
cluster), the streaming attention that reads and updates the ring in one pass, and the layer entry point that chains
them, vs plain FP32 products and the CPU oracle."""
from __future__ import annotations

import pytest
import torch

from oracle import mimi_attention_oracle as O
from test_gpu_layer_blocks import ROUND, _layer_params

pytestmark = pytest.mark.gpu


def _streams(which, T=1):
    """Numbers of live streams either side of where a layer's call of T <= 8 frames takes other kernels: "last", each of whose heads has an SM to itself
    (LayerNorm, projection and attention are one kernel), "next" (two), and "many", more rows than the clusters of 16 blocks could hold that take
    up to 24 each through output projection and MLP (one kernel; for "many" three or four)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {"one": 1, "last": sms // 8, "next": sms // 8 + 1, "many": 24 * (sms // 16) // T + 1}[which]


# rows: one, either side of a tile's edge, two tiles; shapes: every split (8, 4, 2, 1 blocks per cluster) that K and the
# number of tiles lead to, a K that only divides by two, the first size past the rule's edge (two tiles per SM)
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 256, 1100])
@pytest.mark.parametrize("shape", [(512, 512), (2048, 512), (512, 2048), (128, 256), (64, 1536)])
def test_linear_with_few_rows(rows, shape):
    import fast_mimi_b200 as fm
    K, N = shape
    g = torch.Generator(device="cuda").manual_seed(rows * 31 + K)
    a = torch.randn(rows, K, device="cuda", generator=g).half()
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).half()
    s = torch.rand(N, device="cuda", generator=g) + 0.2
    acc = a.double() @ w.double().T
    for out_dtype in (torch.float32, torch.float16):
        r = torch.randn(rows, N, device="cuda", generator=g).to(out_dtype)
        got = fm.ops.linear(a, w, scale=s, residual=r, out_dtype=out_dtype)
        assert O.rel_l2(got.double(), r.double() + s * acc) < max(ROUND[out_dtype], 2e-5)
        got = fm.ops.linear(a, w, activation="gelu", out_dtype=out_dtype)
        assert O.rel_l2(got.double(), torch.nn.functional.gelu(acc)) < max(ROUND[out_dtype], 2e-5)
    fm.check_status()


# K shared out over one, two, four and eight blocks; rows at the edges of tiles of 16, 32 and 64 and of what the kernel takes
@pytest.mark.parametrize("rows,K,N", [(16, 512, 256), (17, 512, 512), (593, 512, 512), (1184, 512, 512), (1185, 512, 512), (2368, 512, 512), (2369, 512, 512),
                                      (33, 1024, 1024), (500, 1024, 512), (128, 1024, 256), (129, 1024, 256), (31, 2048, 512), (33, 2048, 512), (257, 2048, 512), (512, 2048, 512),
                                      (513, 2048, 512), (15, 4096, 512), (65, 4096, 256), (130, 4096, 512), (576, 512, 2048), (577, 512, 2048)])
@pytest.mark.parametrize("in_dtype", [torch.float16, torch.bfloat16])
def test_linear_with_resident_weights(rows, K, N, in_dtype):
    """Products whose weights lie in tensor memory, against 64 bits: FP32 results to 2e-7 (partial sums of at most 128 products, 2^-24 each, and their
    sums), 16-bit ones to their rounding; nothing behind the last row is written."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    a = torch.randn(rows, K, device="cuda", generator=g).to(in_dtype)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(in_dtype)
    s = torch.rand(N, device="cuda", generator=g) + 0.2
    acc = a.double() @ w.double().T
    for out_dtype in (torch.float32, torch.float16, torch.bfloat16):
        r = torch.randn(rows, N, device="cuda", generator=g).to(out_dtype)
        held = torch.full((rows + 1, N), 7.0, dtype=out_dtype, device="cuda")
        fm.ops.linear(a, w, scale=s, residual=r, out_dtype=out_dtype, out=held[:rows])
        taken = K == 512 and (rows <= 2368 and N <= 512 or rows <= 576) or K > 512 and rows <= 512
        bar = {torch.float32: 2e-7 if taken else 2e-6, torch.float16: 5e-4, torch.bfloat16: 4e-3}[out_dtype]
        assert O.rel_l2(held[:rows].double(), r.double() + s * acc) < bar
        assert (held[rows] == 7.0).all()
        got = fm.ops.linear(a, w, activation="gelu", out_dtype=out_dtype)
        assert O.rel_l2(got.double(), torch.nn.functional.gelu(acc)) < max(bar, 2e-6)
    fm.check_status()


# K shared by two, four and eight blocks, rows of 16, 32 and 64 a block: partial sums of the other blocks come where a block's weights lay
@pytest.mark.parametrize("rows,K,N", [(16, 1024, 1024), (300, 1024, 1024), (16, 2048, 512), (64, 2048, 512), (512, 2048, 512), (16, 4096, 256), (60, 4096, 512)])
def test_products_whose_blocks_share_k_repeat_exactly(rows, K, N):
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    a = torch.randn(rows, K, device="cuda", generator=g).half()
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).half()
    first = fm.ops.linear(a, w, out_dtype=torch.float32)
    assert O.rel_l2(first.double(), a.double() @ w.double().T) < 2e-6
    for y in [fm.ops.linear(a, w, out_dtype=torch.float32) for _ in range(100)]:
        assert torch.equal(y, first)
    fm.check_status()


@pytest.mark.parametrize("B,T", [(1, 1), (1, 127), (3, 43), (2, 128), (5, 100)])
def test_projection_with_few_rows(B, T):
    import fast_mimi_b200 as fm
    g = torch.Generator().manual_seed(B * 1000 + T)
    x = torch.randn(B, T, 512, generator=g).bfloat16()
    w = (torch.randn(1536, 512, generator=g) * 0.04).bfloat16()
    pos = torch.randint(0, 3000, (B, T), generator=g)                      # a table per clip
    cos, sin = fm.rope_tables(pos)
    q, k, v = O.qkv_project(x.float(), *w.float().chunk(3, 0))              # [B, 8, T, 64]
    c, s = cos[:, None], sin[:, None]
    rot = lambda t: t * c + O.rotate_half(t) * s
    frames = lambda t: t.transpose(1, 2).reshape(B, T, 512)
    for value_dtype in (torch.float16, torch.bfloat16):
        got = fm.ops.qkv_rope(x.cuda(), w.cuda(), cos.cuda(), sin.cuda(), value_dtype=value_dtype)
        for y, ref, dt in zip(got, (rot(q), rot(k), v), (torch.bfloat16, torch.bfloat16, value_dtype)):
            assert O.rel_l2(y.float().cpu(), frames(ref)) < ROUND[dt]
    fm.check_status()


@pytest.mark.parametrize("window", [250, 100, 3])
@pytest.mark.parametrize("streams", [1, 5, 19])
def test_layer_on_live_streams_matches_the_oracle(streams, window):
    """A session of calls of 1 .. 8 frames (the streaming kernels: one to 18 streams on a B200, 19 and more), longer ones (the tensor-core path) and one beyond the
    window, over rings that fill up and wrap; every call against the oracle's layer on its own cache.  Bar as for the
    layer without a cache: 2e-3 on what the layer adds to its input."""
    import fast_mimi_b200 as fm
    p = _layer_params(70 + window)
    layer = fm.MimiTransformerLayerB200(sliding_window=window).cuda()
    layer.load_state_dict(p, strict=True)
    ring, cache = fm.MimiKVRing(1, streams, window), O.KVCacheOracle(window=window)
    g = torch.Generator().manual_seed(window)
    past = 0
    for T in (1, 1, 2, 7, 60, 1, 8, 7, 200, 3, 1, 7, 260, 1, 2):
        x = torch.randn(streams, T, 512, generator=g)
        cos, sin = fm.rope_tables(torch.arange(past, past + T)[None])
        got, _ = layer(x.cuda(), None, ring, (cos.cuda(), sin.cuda()))
        want = O.transformer_layer(x, p, cache=cache, window=window)
        assert O.rel_l2(got.cpu() - x, want - x) < 2e-3, (T, past)
        past += T
    fm.check_status()


# rings with spare slots, partly filled and wrapped, and one of `window` slots; T: the streaming kernels (two streams and one more than the first of
# them takes), the few-tile kernel with the ring's update inside (a block or, T = 40 of two streams, two of them a stream and head) and
# without, the linearised path (slots > 256, or T = 100 of many streams)
@pytest.mark.parametrize("slots,past", [(256, 150), (256, 300), (250, 90), (120, 500), (100, 400), (300, 350)])
@pytest.mark.parametrize("T", [1, 8, 20, 40, 100])
@pytest.mark.parametrize("streams", ["two", "next"])
def test_slots_outside_the_window_do_not_show(streams, slots, past, T):
    """A layer call over a ring of more slots than the window, non-finite wherever a slot is empty or has left the window:
    output and new rows are those over a ring that holds the window alone.  Bar: the sums run in another order, and a flipped
    rounding of a 16-bit operand is 2^-11 of one value in many."""
    import fast_mimi_b200 as fm
    S, window = 2 if streams == "two" else _streams(streams), 100
    layer = fm.MimiTransformerLayerB200(sliding_window=window).cuda()
    layer.load_state_dict(_layer_params(17))
    g = torch.Generator(device="cuda").manual_seed(past)
    ring = fm.MimiKVRing(1, S, window)
    ring.advance(0, past)
    k = torch.full((S, 8, slots, 64), float("nan"), dtype=torch.bfloat16, device="cuda")
    v = k.half()
    at = torch.arange(past - min(past, window - 1), past, device="cuda")
    for spare, tight in ((k, ring.ring_k[0]), (v, ring.ring_v[0])):
        rows = torch.randn(S, 8, len(at), 64, device="cuda", generator=g).to(spare.dtype)
        spare[:, :, at % slots], tight[:, :, at % window] = rows, rows
    x = torch.randn(S, T, 512, device="cuda", generator=g)
    cs = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])
    want, _ = layer(x, None, ring, cs)
    params, keep = layer._native_plan(x)
    got = fm.ops.layer_forward(params, x, *cs, value_dtype=torch.float16, ring=(k, v), past=past, window=window)
    assert O.rel_l2(got - x, want - x) < 5e-4
    new = torch.arange(max(past, past + T - window), past + T, device="cuda")
    for spare, tight in ((k, ring.ring_k[0]), (v, ring.ring_v[0])):
        assert torch.equal(spare[:, :, new % slots], tight[:, :, new % window])
    fm.check_status()


@pytest.mark.parametrize("value_dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 8])
@pytest.mark.parametrize("streams", ["one", "next"])
def test_streaming_probabilities_keep_the_bits_of_fp32(streams, value_dtype, T):
    """A layer whose output is the attention core of a chosen query over a chosen ring.  FP16 values: all that counts comes
    from probabilities of about 2^-20 beside one of 1 whose value is 0.  BF16 values: +1 and -1 in turn, under probabilities that
    differ by 2^-12 of themselves.  Bar: the result's own rounding; FP32 exponentials (2^-22) add 1e-3 of the BF16 result."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    q, k, v = torch.zeros(8, 64), torch.zeros(8, 250, 64), torch.zeros(8, 250, 64)
    q[:, 0], q[:, 1] = 8.0, 2.0 ** -3                         # logits k_0 + 2^-6 k_1
    with torch.no_grad():
        for p in layer.parameters():
            p.zero_()
        layer.input_layernorm.bias[0] = 1.0
        layer.self_attn.q_proj.weight[:, 0] = q.reshape(-1)
        layer.self_attn.o_proj.weight.copy_(torch.eye(512))
        layer.self_attn_layer_scale.scale.fill_(1.0)
    past = 300
    at = torch.arange(past - 249, past) % 250                 # oldest first; a call of T frames leaves the oldest out one by one
    if value_dtype == torch.float16:
        k[:, at, 0] = (torch.arange(8) / 16)[:, None]
        k[:, at[-1], 0] = 14.0
        v[:, at[:-1]] = 1.0
    else:
        k[:, at, 0] = -torch.tensor([1.0, 1.125, 1.25, 1.5] * 2)[:, None]
        k[:, at[-1], 0] = 0.0
        k[:, at[1:-1:2], 1] = -(2.0 ** -6)
        v[:, at[:-1:2]], v[:, at[1:-1:2]] = 1.0, -1.0
    S = _streams(streams)
    ring = fm.MimiKVRing(1, S, 250, value_dtype=value_dtype)
    ring.ring_k[0], ring.ring_v[0] = k.cuda(), v.cuda()
    assert torch.equal(ring.ring_k[0, 0].float().cpu(), k)
    ring.advance(0, past)
    one = torch.ones(1, T, 64, device="cuda")
    every = layer(torch.zeros(S, T, 512, device="cuda"), None, ring, (one, one * 0))[0].cpu().view(S, T, 8, 64)
    assert torch.equal(every, every[:1].expand_as(every))
    got = every[0]
    new = torch.zeros(8, T, 64)
    kk, vv = torch.cat((k[:, at], new), dim=1).double(), torch.cat((v[:, at], new), dim=1).double()
    for t in range(T):
        s = torch.einsum("hd,hnd->hn", q.double(), kk[:, t:t + 250]) * 0.125
        want = torch.einsum("hn,hnd->hd", torch.softmax(s, dim=-1), vv[:, t:t + 250])
        if value_dtype == torch.float16 or t % 2 == 0:        # else one sign is in the majority, nothing cancels
            assert O.rel_l2(got[t], want) < ROUND[value_dtype], t
    fm.check_status()


@pytest.mark.parametrize("T", [1, 2, 8])
@pytest.mark.parametrize("past", [0, 3, 249, 700])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16)])
def test_a_stream_does_not_depend_on_those_beside_it(T, past, dtype, value_dtype):
    """The kernels that a call takes follow from how many streams share it: what one stream's rows come to must not depend on it but for the order of
    FP32 sums (2^-21 of the branch) and, where that flips the rounding of an operand behind it, 16-bit units (2^-9 BF16, 2^-11 FP16, over 512
    terms with random signs).  Rings are equal bit for bit, and as long as the kernels stay the same so are the results."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    layer.load_state_dict(_layer_params(T + past), strict=True)
    layer = layer.to(dtype)
    g = torch.Generator(device="cuda").manual_seed(past)
    counts = [_streams(which, T) for which in ("many", "next", "last", "one")]
    x = torch.randn(counts[0], T, 512, device="cuda", generator=g).to(dtype)
    cs = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])
    rings = [fm.MimiKVRing(1, n, 250, value_dtype=value_dtype) for n in counts]
    for t in (rings[0].ring_k, rings[0].ring_v):
        t.normal_(generator=g)
    for n, ring in zip(counts[1:], rings[1:]):
        ring.ring_k.copy_(rings[0].ring_k[:, :n])
        ring.ring_v.copy_(rings[0].ring_v[:, :n])
    outs = []
    for n, ring in zip(counts, rings):
        ring.advance(0, past)
        outs.append(layer(x[:n], None, ring, cs)[0])
    for n, ring, y in zip(counts[1:], rings[1:], outs[1:]):
        assert torch.equal(ring.ring_k[0], rings[0].ring_k[0, :n]) and torch.equal(ring.ring_v[0], rings[0].ring_v[0, :n])
        want = outs[0][:n].float() - x[:n].float()
        bound = {torch.float32: 1e-3, torch.float16: 4e-3, torch.bfloat16: 2e-2}[dtype]
        assert O.rel_l2((y.float() - x[:n].float()).cpu(), want.cpu()) < bound
    assert torch.equal(outs[2][:1], outs[3])
    fm.check_status()


@pytest.mark.parametrize("T", [1, 8])
@pytest.mark.parametrize("past", [0, 90, 700])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float16),
                                               (torch.float16, torch.float16)])
def test_live_streams_against_64_bits(T, past, dtype, value_dtype):
    """A layer's call for numbers of streams that take different kernels (``_streams``), from the parameters, the
    rings and the input as they are held, against the same in 64 bits.  FP32 streams: 2e-3 of what the layer adds, the bar of the
    layer without a cache.  16-bit streams are rounded twice on the way (2^-9 BF16, 2^-11 FP16 each at most), which covers
    what the branches add to that.  All routes round alike but for the order of FP32 sums: none is 5 % further off."""
    import fast_mimi_b200 as fm
    window = slots = 250
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    layer.load_state_dict(_layer_params(90 + T + past), strict=True)
    layer = layer.to(dtype).requires_grad_(False)
    g = torch.Generator(device="cuda").manual_seed(past + T)
    counts = [_streams(which, T) for which in ("last", "next", "many")]
    S = counts[0]                                                                    # of every call, those that are looked at
    x = torch.randn(counts[-1], T, 512, device="cuda", generator=g).to(dtype)
    cos, sin = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])
    first = fm.MimiKVRing(1, counts[-1], window, value_dtype=value_dtype)
    for t in (first.ring_k, first.ring_v):
        t.normal_(generator=g)
    held = [t[0, :S].double() for t in (first.ring_k, first.ring_v)]                 # [S, 8, slots, 64]
    got = {}
    for n in counts:
        ring = fm.MimiKVRing(1, n, window, value_dtype=value_dtype)
        ring.ring_k.copy_(first.ring_k[:, :n])
        ring.ring_v.copy_(first.ring_v[:, :n])
        ring.advance(0, past)
        got[n] = layer(x[:n], None, ring, (cos, sin))[0][:S].double()
    p = {k: v.double() for k, v in layer.state_dict().items()}
    xd = x[:S].double()
    norm = lambda t, name: torch.nn.functional.layer_norm(t, (512,), p[name + ".weight"], p[name + ".bias"], 1e-5)
    h = norm(xd, "input_layernorm")
    q, k, v = ((h @ p[f"self_attn.{n}_proj.weight"].T).view(S, T, 8, 64).transpose(1, 2) for n in "qkv")
    turn = lambda t: t * cos.double()[:, None] + O.rotate_half(t) * sin.double()[:, None]
    at = torch.arange(max(0, past - window + 1), past, device="cuda")
    keys, values = torch.cat((held[0][:, :, at % slots], turn(k)), 2), torch.cat((held[1][:, :, at % slots], v), 2)
    pos = torch.cat((at, torch.arange(past, past + T, device="cuda")))
    new = pos[-T:, None]
    seen = (pos[None] <= new) & (pos[None] > new - window)
    core = torch.softmax((turn(q) @ keys.transpose(-1, -2) * 0.125).masked_fill(~seen, float("-inf")), -1) @ values
    x1 = xd + core.transpose(1, 2).reshape(S, T, 512) @ p["self_attn.o_proj.weight"].T * p["self_attn_layer_scale.scale"]
    y = x1 + torch.nn.functional.gelu(norm(x1, "post_attention_layernorm") @ p["mlp.fc1.weight"].T) @ p["mlp.fc2.weight"].T * p["mlp_layer_scale.scale"]
    base = xd if dtype == torch.float32 else torch.zeros_like(xd)
    off = {n: O.rel_l2(got[n] - base, y - base) for n in got}
    assert max(off.values()) < {torch.float32: 2e-3, torch.bfloat16: 2 ** -8, torch.float16: 2 ** -10}[dtype], off
    assert max(off.values()) < 1.05 * min(off.values()), off
    fm.check_status()


@pytest.mark.parametrize("past", [0, 20, 249, 400])
@pytest.mark.parametrize("T", [9, 32, 33, 64, 65])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.bfloat16, torch.bfloat16)])
def test_chunks_of_few_streams_in_blocks_of_32_and_64_queries(T, past, dtype, value_dtype):
    """Five streams' chunks take blocks of 32 queries (two of them, with up to 64 frames, share a ring and update it together), forty take 64 or other
    kernels: rings are equal bit for bit, what a layer adds agrees but for the order of FP32 sums, i.e. where that flips the rounding of a
    16-bit operand (bounds as above)."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    layer.load_state_dict(_layer_params(T + past), strict=True)
    layer = layer.to(dtype)
    g = torch.Generator(device="cuda").manual_seed(past + T)
    x = torch.randn(40, T, 512, device="cuda", generator=g).to(dtype)
    cs = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])
    many, few = fm.MimiKVRing(1, 40, 250, value_dtype=value_dtype), fm.MimiKVRing(1, 5, 250, value_dtype=value_dtype)
    for t, u in ((many.ring_k, few.ring_k), (many.ring_v, few.ring_v)):
        t.normal_(generator=g)
        u.copy_(t[:, :5])
    for ring in (many, few):
        ring.advance(0, past)
    want, got, base = layer(x, None, many, cs)[0][:5].float(), layer(x[:5], None, few, cs)[0].float(), x[:5].float()
    assert O.rel_l2((got - base).cpu(), (want - base).cpu()) < {torch.float32: 1e-3, torch.bfloat16: 2e-2}[dtype]
    assert torch.equal(few.ring_k, many.ring_k[:, :5]) and torch.equal(few.ring_v, many.ring_v[:, :5])
    fm.check_status()


# rows of the larger call: 480 (LayerNorm inside the projection), 800, 1000 and 1024 (weights resident in tensor memory), 1025 and 1280 (the few-row kernel),
# 2400 (pairs of blocks); of the smaller one: 20 to 600
@pytest.mark.parametrize("streams,T", [(24, 20), (40, 20), (40, 25), (32, 32), (1024, 1), (1025, 1), (64, 20), (60, 40)])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.bfloat16, torch.bfloat16)])
def test_a_ring_does_not_depend_on_the_streams_beside_it(streams, T, dtype, value_dtype):
    """What a layer's call writes into a stream's ring is the same bit for bit however many other streams share the call, i.e. whichever kernel
    makes k and v: each sums K = 512 in one accumulator."""
    import fast_mimi_b200 as fm
    past = 300
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    layer.load_state_dict(_layer_params(T), strict=True)
    layer = layer.to(dtype)
    g = torch.Generator(device="cuda").manual_seed(streams)
    x = torch.randn(streams, T, 512, device="cuda", generator=g).to(dtype)
    cs = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])

    def rings(n):
        ring = fm.MimiKVRing(1, n, 250, value_dtype=value_dtype)
        ring.advance(0, past)
        layer(x[:n], None, ring, cs)
        return ring.ring_k[0], ring.ring_v[0]

    whole = rings(streams)
    for n in (1, 15 if T > 8 else 600):
        for few, many in zip(rings(n), whole):
            assert torch.equal(few, many[:n])
    fm.check_status()


# past: nothing, either side of a warp's sixteen slots, of a full ring and of its turn; 18 streams are the last that take the kernel on a B200
@pytest.mark.parametrize("past", [0, 1, 15, 16, 17, 241, 249, 250, 257, 1000])
@pytest.mark.parametrize("streams,T", [(1, 1), (2, 3), (18, 8)])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16)])
def test_first_half_of_a_call_for_few_streams(streams, T, past, dtype, value_dtype):
    """LayerNorm, projection and attention as one kernel (up to 18 streams) and as two (the same streams among 19): rings are equal bit
    for bit, what a layer adds agrees but for the order of FP32 sums, i.e. where that flips the rounding of a 16-bit operand (bounds as
    in ``test_a_stream_does_not_depend_on_those_beside_it``)."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(value_dtype=value_dtype).cuda()
    layer.load_state_dict(_layer_params(T + past), strict=True)
    layer = layer.to(dtype)
    g = torch.Generator(device="cuda").manual_seed(past + T)
    x = torch.randn(19, T, 512, device="cuda", generator=g).to(dtype)
    cs = fm.rope_tables(torch.randint(0, 3000, (19, T), device="cuda", generator=g))           # a table per stream
    many, few = fm.MimiKVRing(1, 19, 250, value_dtype=value_dtype), fm.MimiKVRing(1, streams, 250, value_dtype=value_dtype)
    for t, u in ((many.ring_k, few.ring_k), (many.ring_v, few.ring_v)):
        t.normal_(generator=g)
        u.copy_(t[:, :streams])
    for ring in (many, few):
        ring.advance(0, past)
    want = layer(x, None, many, cs)[0][:streams].float()
    got = layer(x[:streams], None, few, tuple(t[:streams] for t in cs))[0].float()
    base = x[:streams].float()
    bound = {torch.float32: 1e-3, torch.float16: 4e-3, torch.bfloat16: 2e-2}[dtype]
    assert O.rel_l2((got - base).cpu(), (want - base).cpu()) < bound
    assert torch.equal(few.ring_k, many.ring_k[:, :streams]) and torch.equal(few.ring_v, many.ring_v[:, :streams])
    fm.check_status()


# rows: one, either side of a cluster's rows (8) and of what seven clusters of 8, 16 and 24 rows hold; of where LayerNorm's products go from 16 to 32
# and 64 rows a block (96, 192), of the last that have LayerNorm inside (576 and 768) and of those whose second MLP product has blocks of 128 rows (513 .. 1024); an MLP of another size, for which fewer kernels are there
@pytest.mark.parametrize("B,T,ffn", [(1, 1, 2048), (1, 8, 2048), (1, 9, 2048), (1, 56, 2048), (1, 57, 2048), (1, 112, 2048), (1, 113, 2048), (2, 61, 2048),
                                     (1, 96, 2048), (1, 97, 2048), (1, 168, 2048), (1, 169, 2048), (1, 193, 2048), (3, 192, 2048), (1, 513, 2048),
                                     (1, 577, 2048), (3, 256, 2048), (1, 769, 2048), (2, 512, 2048), (1, 1025, 2048), (1, 9, 1024)])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float32, torch.float16), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16),
                                               (torch.bfloat16, torch.float16), (torch.float16, torch.float16)])
def test_layer_on_few_rows_against_64_bits(B, T, ffn, dtype, value_dtype):
    """A layer on clips of few rows in all, against the same in 64 bits; bars as for
    live streams below (BF16 values: their rounding, 2^-9, in front of the output projection)."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(intermediate_size=ffn, value_dtype=value_dtype).cuda()
    p = _layer_params(T)
    p["mlp.fc1.weight"], p["mlp.fc2.weight"] = p["mlp.fc1.weight"][:ffn].contiguous(), p["mlp.fc2.weight"][:, :ffn].contiguous()
    layer.load_state_dict(p, strict=True)
    layer = layer.to(dtype).requires_grad_(False)
    g = torch.Generator(device="cuda").manual_seed(B * T)
    x = torch.randn(B, T, 512, device="cuda", generator=g).to(dtype)
    cos, sin = fm.rope_tables(torch.arange(T, device="cuda")[None])
    y = layer(x, None, None, (cos, sin))[0]
    p = {k: v.double() for k, v in layer.state_dict().items()}
    xd = x.double()
    norm = lambda t, name: torch.nn.functional.layer_norm(t, (512,), p[name + ".weight"], p[name + ".bias"], 1e-5)
    q, k, v = ((norm(xd, "input_layernorm") @ p[f"self_attn.{n}_proj.weight"].T).view(B, T, 8, 64).transpose(1, 2) for n in "qkv")
    turn = lambda t: t * cos.double()[:, None] + O.rotate_half(t) * sin.double()[:, None]
    ones = torch.ones(T, T, dtype=torch.bool, device="cuda")
    hidden = ones.triu(1) | ones.tril(-250)
    core = torch.softmax((turn(q) @ turn(k).transpose(-1, -2) * 0.125).masked_fill(hidden, float("-inf")), -1) @ v
    x1 = xd + core.transpose(1, 2).reshape(B, T, 512) @ p["self_attn.o_proj.weight"].T * p["self_attn_layer_scale.scale"]
    want = x1 + torch.nn.functional.gelu(norm(x1, "post_attention_layernorm") @ p["mlp.fc1.weight"].T) @ p["mlp.fc2.weight"].T * p["mlp_layer_scale.scale"]
    base = xd if dtype == torch.float32 else torch.zeros_like(xd)
    bar = {torch.float32: 2e-3 if value_dtype == torch.float16 else 4e-3, torch.bfloat16: 2 ** -8, torch.float16: 2 ** -10}[dtype]
    assert O.rel_l2(y.double() - base, want - base) < bar
    fm.check_status()


# rows of the larger call: 200 and 500 (LayerNorm inside the product), 600, 640 and 768 (weights resident in tensor memory); of the smaller one: 8 to 100, for which
# the MLP is part of one kernel with 8, 16 or 24 rows a cluster (8 to 56, to 112, to 168 rows)
@pytest.mark.parametrize("clips,T,few", [(2, 100, 1), (5, 100, 1), (6, 100, 1), (8, 96, 1), (96, 8, 1), (10, 60, 1), (4, 160, 1), (10, 60, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_hidden_units_do_not_depend_on_the_clips_beside_them(clips, T, few, dtype):
    """What fc1 and GELU make of a frame is the same bit for bit in every kernel that takes up to 768 rows: each sums 256 of K = 512 in an accumulator.
    W_o = 0 and rows of the identity as W_2, so that a layer adds 512 of its hidden units, or the last 512, to its input."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200().cuda()
    layer.load_state_dict(_layer_params(T), strict=True)
    with torch.no_grad():
        layer.self_attn.o_proj.weight.zero_()
        layer.mlp_layer_scale.scale.fill_(1.0)
    layer = layer.to(dtype).requires_grad_(False)
    x = torch.randn(clips, T, 512, device="cuda", generator=torch.Generator(device="cuda").manual_seed(clips)).to(dtype)
    cs = fm.rope_tables(torch.arange(T, device="cuda")[None])
    for unit in (0, 2048 - 512):
        layer.mlp.fc2.weight.zero_()
        layer.mlp.fc2.weight[:, unit:unit + 512].fill_diagonal_(1.0)
        assert torch.equal(layer(x[:few], None, None, cs)[0], layer(x, None, None, cs)[0][:few])
    fm.check_status()


@pytest.mark.parametrize("T", [1, 8])
@pytest.mark.parametrize("which", ["one", "last", "next", "many"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_live_streams_without_layer_scales(which, T, dtype):
    """The native call takes a layer without scales (NULL) as one whose scales are one, bit for bit, whichever kernels apply
    them, and refuses scales off a 16-byte boundary."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200().cuda()
    layer.load_state_dict(_layer_params(31), strict=True)
    layer = layer.to(dtype).requires_grad_(False)
    layer.self_attn_layer_scale.scale.fill_(1.0)
    layer.mlp_layer_scale.scale.fill_(1.0)
    streams = _streams(which, T)
    g = torch.Generator(device="cuda").manual_seed(streams + T)
    x = torch.randn(streams, T, 512, device="cuda", generator=g).to(dtype)
    past = 40
    cos, sin = fm.rope_tables(torch.arange(past, past + T, device="cuda")[None])
    ring = fm.MimiKVRing(1, streams, 250)
    for t in (ring.ring_k, ring.ring_v):
        t.normal_(generator=g)
    params, keep = layer._native_plan(x)
    one_k, one_v = ring.ring_k[0].clone(), ring.ring_v[0].clone()
    call = lambda k, v: fm.ops.layer_forward(params, x, cos, sin, value_dtype=torch.float16, ring=(k, v), past=past, window=250)
    ones = call(one_k, one_v)
    scale = params.attn_scale
    params.attn_scale = scale + x.element_size()
    with pytest.raises(RuntimeError, match="misaligned"):
        call(ring.ring_k[0].clone(), ring.ring_v[0].clone())
    params.attn_scale = params.mlp_scale = None
    null_k, null_v = ring.ring_k[0].clone(), ring.ring_v[0].clone()
    assert torch.equal(call(null_k, null_v), ones)
    assert torch.equal(null_k, one_k) and torch.equal(null_v, one_v)
    fm.check_status()


def test_layer_follows_its_ring():
    """A session whose ring goes through pickle, then gets new storage, half way: outputs and rings are those of a session
    left alone."""
    import pickle
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200(layer_idx=1).cuda()
    plain, other = fm.MimiKVRing(2, 2, 250), fm.MimiKVRing(2, 2, 250)
    x = torch.randn(4, 2, 1, 512, device="cuda")
    for i in range(4):
        if i == 2:
            other = pickle.loads(pickle.dumps(other))
        elif i == 3:
            other.ring_k.data, other.ring_v.data = other.ring_k.clone(), other.ring_v.clone()
        cs = fm.rope_tables(torch.tensor([[i]], device="cuda"))
        a, b = layer(x[i], None, plain, cs)[0], layer(x[i], None, other, cs)[0]
        assert torch.equal(a, b)
        for s, t in zip(plain.ordered(1), other.ordered(1)):
            assert torch.equal(s, t)
    fm.check_status()


@pytest.mark.parametrize("stream_dtype", [torch.float32, torch.bfloat16])
def test_live_streams_with_bf16_values_and_tables_of_their_own(stream_dtype):
    """BF16 values in the ring (streaming, few-tile and linearised attention) under rotary tables that differ by stream: each
    stream's positions start elsewhere, which a rotation applied to q and k alike does not show.  Bar: BF16 roundings of
    values, probabilities, core and W_o (2^-9 / sqrt 3 each, 2.3e-3 in quadrature), of the LayerNorms' results and the MLP's inner
    values too in a BF16 stream (8e-3), plus that stream's own two roundings."""
    import fast_mimi_b200 as fm
    p = {k: v.to(stream_dtype) for k, v in _layer_params(33).items()}
    layer = fm.MimiTransformerLayerB200(value_dtype=torch.bfloat16).cuda().to(stream_dtype)
    layer.load_state_dict(p)
    p = {k: v.float() for k, v in p.items()}
    streams = 3
    starts = torch.tensor([0, 40, 1000])
    ring, cache = fm.MimiKVRing(1, streams, 250, value_dtype=torch.bfloat16), O.KVCacheOracle()
    g = torch.Generator().manual_seed(33)
    past = 0
    for T in (1, 3, 8, 60, 230, 1, 8, 20, 70, 300, 1):
        x = torch.randn(streams, T, 512, generator=g).to(stream_dtype)
        cos, sin = fm.rope_tables(starts[:, None] + torch.arange(past, past + T)[None])
        got, _ = layer(x.cuda(), None, ring, (cos.cuda(), sin.cuda()))
        want = O.transformer_layer(x.float(), p, cache=cache) - x.float()
        bar = ROUND[torch.bfloat16]
        if stream_dtype == torch.bfloat16:
            bar = 8e-3 + 2.0 ** -9 * float((want + x.float()).norm() / want.norm())
        assert O.rel_l2(got.float().cpu() - x.float(), want) < bar, (T, past)
        past += T
    fm.check_status()


@pytest.mark.parametrize("value_dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,window", [(400, 300), (400, 257), (65, 64), (64, 1000), (1, 300)])
def test_one_clip_with_windows_of_any_length(T, window, value_dtype):
    """The few-tile kernel without a ring, also for windows that no ring has."""
    import fast_mimi_b200 as fm
    p = _layer_params(35)
    layer = fm.MimiTransformerLayerB200(sliding_window=window, value_dtype=value_dtype).cuda()
    layer.load_state_dict(p)
    x = torch.randn(1, T, 512, generator=torch.Generator().manual_seed(T))
    cos, sin = fm.rope_tables(torch.arange(T)[None])
    got, _ = layer(x.cuda(), None, None, (cos.cuda(), sin.cuda()))
    want = O.transformer_layer(x, p, window=window)
    assert O.rel_l2(got.cpu() - x, want - x) < max(2e-3, ROUND[value_dtype])
    fm.check_status()


@pytest.mark.parametrize("module,ring", [(torch.float16, torch.bfloat16), (torch.bfloat16, torch.float16)])
def test_layer_on_a_ring_of_the_other_value_type(module, ring):
    """The ring decides the type its values have, whatever the module was built with.  Bar: one BF16 rounding each of values,
    probabilities, result and W_o at most (2^-9 / sqrt 3 of their size), in quadrature 2.3e-3."""
    import fast_mimi_b200 as fm
    p = _layer_params(31)
    layer = fm.MimiTransformerLayerB200(value_dtype=module).cuda()
    layer.load_state_dict(p)
    cache, ref = fm.MimiKVRing(1, 2, 250, value_dtype=ring), O.KVCacheOracle()
    g = torch.Generator().manual_seed(31)
    past = 0
    for T in (1, 5, 240, 1, 30):
        x = torch.randn(2, T, 512, generator=g)
        cos, sin = fm.rope_tables(torch.arange(past, past + T)[None])
        got, _ = layer(x.cuda(), None, cache, (cos.cuda(), sin.cuda()))
        want = O.transformer_layer(x, p, cache=ref)
        assert O.rel_l2(got.cpu() - x, want - x) < ROUND[torch.bfloat16], (T, past)
        past += T
        assert cache.get_seq_length(0) == past
    fm.check_status()


def test_layer_follows_its_parameters():
    """The layer's parameter block is rebuilt when a parameter is written to, replaced, or the options change."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200().cuda()
    x = torch.randn(1, 20, 512, device="cuda")
    cs = fm.rope_tables(torch.arange(20, device="cuda")[None])
    run = lambda: layer(x, None, None, cs)[0]
    for p in (_layer_params(1), _layer_params(2)):
        layer.load_state_dict(p)
        assert O.rel_l2(run().cpu() - x.cpu(), O.transformer_layer(x.cpu(), p) - x.cpu()) < 2e-3
    adds = lambda **kw: O.transformer_layer(x.cpu(), {k: v.cpu() for k, v in layer.state_dict().items()}, **kw) - x.cpu()
    old = adds()
    layer.mlp.fc2 = torch.nn.Linear(2048, 512, bias=False).cuda().requires_grad_(False)
    assert O.rel_l2(run().cpu() - x.cpu(), adds()) < 2e-3 < O.rel_l2(old, adds()) / 4
    old = adds()
    layer.self_attn.sliding_window = 4
    assert O.rel_l2(run().cpu() - x.cpu(), adds(window=4)) < 2e-3 < O.rel_l2(old, adds(window=4)) / 4


def test_layer_follows_an_assigned_data():
    """Two assignments of ``.data`` in a row give a parameter the memory of its first storage again.  The new values have the
    size of the old ones (larger q and LayerNorm weights sharpen the softmax and magnify the rounding of its scores), so the bar
    is that of the layer's other tests."""
    import fast_mimi_b200 as fm
    p = _layer_params(8)
    layer = fm.MimiTransformerLayerB200().cuda()
    layer.load_state_dict(p)
    x = torch.randn(1, 20, 512)
    cs = fm.rope_tables(torch.arange(20, device="cuda")[None])
    layer(x.cuda(), None, None, cs)
    came_back = 0
    for name in ("mlp.fc1.weight", "mlp.fc2.weight", "self_attn.q_proj.weight", "self_attn.o_proj.weight", "input_layernorm.weight"):
        w = layer.get_parameter(name)
        at, a, b = w.data_ptr(), p[name] * 0.5, -p[name]
        w.data = a.cuda()
        w.data = b.cuda()
        came_back += w.data_ptr() == at
        p[name] = b
        got, _ = layer(x.cuda(), None, None, cs)
        assert O.rel_l2(got.cpu() - x, O.transformer_layer(x, p) - x) < 2e-3, name
    assert came_back > 0           # else the allocator has changed and this shows nothing


@pytest.mark.parametrize("streams", [38, 64, 333, 700])
def test_many_streams_repeat_exactly(streams):
    """More (stream, head) items than two per SM: three ring slices are in flight per block and its two groups of warps take
    them in turn.  Which slice lands first must not matter: the same call repeats bit for bit, and its first and last streams
    are those of a call by themselves (one item per block)."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(streams)
    w = (torch.randn(1536, 512, device="cuda", generator=g) * 0.04).bfloat16()
    x = torch.randn(streams, 512, device="cuda", generator=g).bfloat16()
    ring_k = torch.randn(streams, 8, 250, 64, device="cuda", generator=g).bfloat16()
    ring_v = torch.randn(streams, 8, 250, 64, device="cuda", generator=g).half()
    layer = fm.MimiTransformerLayerB200().cuda()
    cos, sin = fm.rope_tables(torch.arange(700, 701, device="cuda")[None])
    some = [0, 1, streams - 1]

    def step(rows):
        k, v = ring_k[rows].clone(), ring_v[rows].clone()
        return fm.ops.decode_step(x[rows].contiguous(), w, cos, sin, k, v, 700), k, v

    def whole(rows):
        ring = fm.MimiKVRing(1, len(rows), 250)
        ring.ring_k.copy_(ring_k[rows][None])
        ring.ring_v.copy_(ring_v[rows][None])
        ring.advance(0, 700)
        return layer(x[rows].float()[:, None], None, ring, (cos, sin))[0], ring.ring_k[0], ring.ring_v[0]

    every = list(range(streams))
    for call, bar in ((step, 1e-3), (whole, 1e-4)):
        first = call(every)
        for _ in range(20):
            for a, b in zip(call(every), first):
                assert torch.equal(a, b)
        for a, b in zip(call(some), first):
            assert O.rel_l2(a.double(), b[some].double()) < bar            # other splits of K: FP32 sums in another order
    fm.check_status()


def test_layer_on_half_a_million_streams():
    """A ring's size, not the number of streams, is what the streaming kernel is limited by.  Bar as above: K in other splits."""
    import fast_mimi_b200 as fm
    streams, some = (1 << 19) + 1, [0, 1, 1 << 19]
    layer = fm.MimiTransformerLayerB200(sliding_window=2).cuda()
    ring, few = fm.MimiKVRing(1, streams, 2), fm.MimiKVRing(1, len(some), 2)
    for past in range(3):
        x = torch.randn(streams, 1, 512, device="cuda")
        cs = fm.rope_tables(torch.tensor([[past]], device="cuda"))
        a, b = layer(x, None, ring, cs)[0][some], layer(x[some], None, few, cs)[0]
        assert O.rel_l2(a - x[some], b - x[some]) < 1e-3
    fm.check_status()


def test_layer_with_parameters_that_cannot_be_watched():
    """LayerNorm parameters made in inference mode have no version counter: the call works without a plan."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200().cuda()
    p = _layer_params(4)
    layer.load_state_dict(p)
    with torch.inference_mode():
        layer.input_layernorm.weight = torch.nn.Parameter(p["input_layernorm.weight"].cuda(), requires_grad=False)
    x = torch.randn(1, 20, 512)
    cs = fm.rope_tables(torch.arange(20, device="cuda")[None])
    for _ in range(2):
        got, _ = layer(x.cuda(), None, None, cs)
        assert O.rel_l2(got.cpu() - x, O.transformer_layer(x, p) - x) < 2e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [20, 400, 5000])
def test_layer_reads_its_vectors_where_they_lie(dtype, rows):
    """LayerNorm parameters and layer scales written through ``.data`` (no version counter moves) show in the next call: with
    the LayerNorm folded into the products, with both kinds of linear kernel behind a LayerNorm kernel, and for a module
    whose vectors have several types.  Bars on what the layer adds to its input: 4.5e-3 (the 2e-3 of the other tests times
    1.5^2: larger LayerNorm weights make the scores, and the rounding of q and k in them, so much larger), 8e-3 where the operands
    are BF16, and for a 16-bit stream its two roundings (2^-12 or 2^-9 of its size).  What the old values would give misses them."""
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200().cuda()
    layer.load_state_dict(_layer_params(5))
    layer = layer.to(dtype)
    T = min(rows, 500)
    x = torch.randn(rows // T, T, 512).to(dtype)
    cs = fm.rope_tables(torch.arange(T, device="cuda")[None])

    def wanted():
        return O.transformer_layer(x.float(), {k: v.float().cpu() for k, v in layer.state_dict().items()}) - x.float()

    def check(old=None):
        want = wanted()
        rounding = {torch.float32: 0.0, torch.float16: 2.0 ** -12, torch.bfloat16: 2.0 ** -9}[x.dtype]
        bar = (8e-3 if x.dtype == torch.bfloat16 else 4.5e-3) + rounding * float((want + x.float()).norm() / want.norm())
        got, _ = layer(x.cuda(), None, None, cs)
        assert O.rel_l2(got.float().cpu() - x.float(), want) < bar
        if old is not None:
            assert O.rel_l2(old, want) > 4 * bar
        return want

    ln1, ln2 = layer.input_layernorm, layer.post_attention_layernorm
    scales = layer.self_attn_layer_scale.scale, layer.mlp_layer_scale.scale
    writes = [lambda: ln1.weight.data.mul_(1.5), lambda: ln2.weight.data.mul_(1.5), lambda: ln1.bias.data.add_(0.25),
              lambda: ln2.bias.data.add_(0.25), lambda: scales[0].data.mul_(3.0), lambda: scales[1].data.mul_(-2.0)]
    with torch.no_grad():
        old = check()
        if rows == 20:                                 # one by one
            for write in writes:
                write()
                old = check(old)
        else:
            for write in writes:
                write()
            old = check(old)
        ln1.float()
        old = check()
        ln1.weight.data.mul_(0.5)
        check(old)
        layer = layer.to(torch.bfloat16)               # a 16-bit module in an FP32 stream
        ln1.weight.data.mul_(2.0)
        x = x.float()
        old = check()
        ln1.weight.data.mul_(0.5)
        check(old)
        x = x.half()                                   # and in a stream of the other 16-bit type
        old = check()
        ln1.weight.data.mul_(2.0)
        check(old)
    fm.check_status()


def test_objects_without_what_is_kept_between_calls():
    """Layers, rings and quantisers that were pickled before they kept anything between calls lack those attributes."""
    import fast_mimi_b200 as fm

    def stripped(made, names):
        old = type(made).__new__(type(made))
        old.__dict__.update({k: v for k, v in made.__dict__.items() if k not in names})
        return old

    layer, ring = fm.MimiTransformerLayerB200().cuda(), fm.MimiKVRing(1, 1, 250)
    old, old_ring = stripped(layer, {"_plan"}), stripped(fm.MimiKVRing(1, 1, 250), {"_rings"})
    old.self_attn = stripped(layer.self_attn, {"_packed_from", "_wo16_from", "_packed", "_wo16"})
    old.self_attn._packed = old.self_attn._wo16 = None
    x, cs = torch.randn(1, 20, 512, device="cuda"), fm.rope_tables(torch.arange(20, device="cuda")[None])
    assert torch.equal(old(x, None, old_ring, cs)[0], layer(x, None, ring, cs)[0])
    branch = lambda: fm.MimiRVQB200(torch.randn(1, 2048, 256, device="cuda"), torch.randn(256, 512, 1, device="cuda"),
                                    torch.randn(512, 256, 1, device="cuda"))
    split = fm.MimiSplitRVQB200(branch(), branch())
    old = stripped(split, {"_joint", "_joint_in"})
    e = torch.randn(1, 512, 5, device="cuda")
    codes = split.encode(e)
    assert torch.equal(old.encode(e), codes) and torch.equal(old.decode(codes), split.decode(codes))


# one to three steps a block (a converting pass in front), four of short sequences (as well), then inside: five (a sequence each), six (two
# sequences), seven and eight (shares that run on from one sequence into the next)
@pytest.mark.parametrize("B,T,window", [(1, 257, 250), (2, 384, 130), (1, 385, 257), (3, 640, 250), (5, 1001, 249), (20, 300, 250),
                                        (18, 513, 130), (37, 300, 249), (19, 700, 257), (45, 260, 250)])
@pytest.mark.parametrize("value_dtype", [torch.float16, torch.bfloat16])
def test_fp32_tensors_of_any_layout_in_long_clips(B, T, window, value_dtype):
    """FP32 q, k, v of calls with some steps a block are rounded inside the attention kernel.  The rounding is that of the converting pass, which tensors with a
    stride that a tensor map cannot have (a clip repeated by expand) still take: equal bit for bit.  Shares of a block begin and
    end anywhere in a sequence.  Bound: q and k in BF16 (2^-9 each, over sqrt(64) terms), v and probabilities in 16 bit."""
    from fast_mimi_b200 import ops
    torch.manual_seed(T + window)
    layouts = [lambda: torch.randn(B, T, 8, 64, device="cuda").transpose(1, 2), lambda: torch.randn(B, 8, T, 64, device="cuda"),
               lambda: torch.randn(T, B, 8, 72, device="cuda")[..., :64].permute(1, 2, 0, 3),
               lambda: torch.randn(B, T, 3, 8, 64, device="cuda")[:, :, 1].transpose(1, 2)]
    q, k, v = layouts[0](), layouts[1](), layouts[2]()
    y = ops.window_attention(q, k, v, window=window, value_dtype=value_dtype)
    again = ops.window_attention(*(t.clone(memory_format=torch.contiguous_format) for t in (q, k, v)), window=window, value_dtype=value_dtype)
    assert torch.equal(y, again)
    for b in {0, B - 1}:
        twice = ops.window_attention(*(t[b:b + 1].expand(2, -1, -1, -1) for t in (q, k, v)), window=window, value_dtype=value_dtype)
        assert torch.equal(twice[0], y[b]) and torch.equal(twice[1], y[b])
    q, k, v = (layouts[3]() for _ in range(3))
    y = ops.window_attention(q, k, v, window=window, value_dtype=value_dtype)
    i = torch.arange(T, device="cuda")
    seen = (i[None] <= i[:, None]) & (i[None] > i[:, None] - window)
    ref = torch.softmax((q.double() @ k.double().transpose(-1, -2) * 0.125).masked_fill(~seen, float("-inf")), -1) @ v.double()
    assert O.rel_l2(y.double().cpu(), ref.cpu()) < (8e-3 if value_dtype == torch.float16 else 1e-2)


# Steps a block as above: three; four of a sequence each, of shares that run on through long sequences, through short ones; five and six of the
# latter; six of whole sequences.
@pytest.mark.parametrize("B,T,inside", [(18, 257, False), (16, 385, True), (12, 700, True), (24, 300, False), (21, 385, False), (22, 513, True), (37, 257, True)])
def test_fp32_tensors_are_converted_where_that_is_faster(B, T, inside):
    """The workspaces are written by the converting pass alone.  (Measured, in front and inside: 18.2 and 18.2 us, 23.3 and 22.5, 29.5 and 27.3,
    25.0 and 27.6, 30.7 and 31.7, 41.2 and 37.4, 35.1 and 30.9.)"""
    import ctypes
    from fast_mimi_b200 import _native
    q, k, v = (torch.randn(B, T, 512, device="cuda") for _ in range(3))
    ws = [torch.full((B, T, 512), -7.0, device="cuda", dtype=torch.float16) for _ in range(3)]
    out = torch.empty(B, T, 512, device="cuda")
    strides = (ctypes.c_longlong * 9)(*[T * 512, 64, 512] * 3)
    rc = _native.load().fm_window_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), 2, strides, *(w.data_ptr() for w in ws), None, out.data_ptr(), B, T, 250,
                                            0.125, 1, None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and all(bool((w == -7.0).all()) == inside for w in ws)


# rows: either side of what blocks of 16, 32 and 64 hold at once, and of a last block of one row
@pytest.mark.parametrize("rows", [1, 16, 17, 192, 193, 384, 385, 768, 769])
@pytest.mark.parametrize("dtype,value_dtype", [(torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16), (torch.float16, torch.bfloat16)])
def test_projection_of_few_rows_against_64_bits(rows, dtype, value_dtype):
    """q, k and v of few rows with RoPE against 64 bits.  A value is off by its rounding at most, BF16 for q and k, and by FP32 sums of
    512 products, nothing beside it: in the mean of squares less than half a unit of the last place, 2^-9 and 2^-12."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(1, rows, 512, device="cuda", generator=g).to(dtype)
    w = (torch.randn(1536, 512, device="cuda", generator=g) * 0.03).to(dtype)
    cos, sin = fm.rope_tables(torch.arange(rows, device="cuda")[None])
    got = fm.ops.qkv_rope(x, w, cos, sin, value_dtype=value_dtype)
    want = (x[0].double() @ w.double().T).view(rows, 3, 8, 64)
    for i, (t, bar) in enumerate(zip(got, (2 ** -9, 2 ** -9, 2 ** -12 if value_dtype == torch.float16 else 2 ** -9))):
        e = want[:, i]
        if i < 2:
            e = e * cos[0].double()[:, None] + O.rotate_half(e) * sin[0].double()[:, None]
        assert O.rel_l2(t.view(rows, 8, 64).double(), e) < bar
    fm.check_status()


@pytest.mark.parametrize("call", ["streams", "clip", "clips", "linear", "attention", "window", "encode", "decode", "downsample"])
def test_a_call_may_be_its_threads_first(call):
    """Threads that have made no CUDA call yet and whose memory comes out of the allocator's pool: no context is bound to them.  Results are those of
    the thread that made the objects."""
    import threading
    import types
    import fast_mimi_b200 as fm
    torch.manual_seed(0)
    cs = lambda T: fm.rope_tables(torch.arange(T, device="cuda")[None])
    if call in ("streams", "clip", "clips"):
        layer = fm.MimiTransformerLayerB200().cuda()
        layer.load_state_dict(_layer_params(3))
        S, T = {"streams": (3, 1), "clip": (1, 125), "clips": (5, 100)}[call]
        x, tables = torch.randn(S, T, 512, device="cuda"), cs(T)
        ring = fm.MimiKVRing(1, S, 250) if call == "streams" else None

        def run():
            if ring is not None:
                ring.reset()
            return layer(x, None, ring, tables)[0]
    elif call == "linear":
        a, w = torch.randn(200, 512, device="cuda").half(), torch.randn(512, 512, device="cuda").half()
        run = lambda: fm.ops.linear(a, w, out_dtype=torch.float32)
    elif call == "attention":
        x, w, tables = torch.randn(2, 200, 512, device="cuda").bfloat16(), (torch.randn(1536, 512, device="cuda") * 0.02).bfloat16(), cs(200)
        run = lambda: fm.ops.attention_prefill(x, w, *tables)
    elif call == "window":
        q, k, v = (torch.randn(1, 400, 8, 64, device="cuda").half().transpose(1, 2) for _ in range(3))
        run = lambda: fm.native_window_attention(q, k, v, scale=0.125, window=250)
    elif call in ("encode", "decode"):
        branch = lambda n: fm.MimiRVQB200(torch.randn(n, 2048, 256, device="cuda"), torch.randn(256, 512, 1, device="cuda"),
                                          torch.randn(512, 256, 1, device="cuda"))
        split = fm.MimiSplitRVQB200(branch(1), branch(7))
        e = torch.randn(1, 512, 1, device="cuda")               # one frame: nothing to lay out anew in front
        codes = split.encode(e)
        run = (lambda: split.encode(e)) if call == "encode" else (lambda: split.decode(codes))
    else:
        conv = torch.nn.Conv1d(512, 512, 4, 2, bias=False, device="cuda").requires_grad_(False)
        down = fm.MimiDownsampleB200(types.SimpleNamespace(conv=conv, causal=True, pad_mode="replicate"))
        e = torch.randn(1, 125, 512, device="cuda").transpose(1, 2)
        run = lambda: down(e)
    with torch.no_grad():
        want = run()
        run()                                                   # its result goes back to the pool
        torch.cuda.synchronize()
        for _ in range(2):
            got = []

            def body():
                with torch.no_grad():
                    try:
                        got.append(run())
                    except Exception as error:                  # noqa: BLE001
                        got.append(error)

            thread = threading.Thread(target=body)
            thread.start()
            thread.join()
            assert isinstance(got[0], torch.Tensor), got[0]
            torch.cuda.synchronize()
            assert torch.equal(got[0], want)
            got.clear()
    fm.check_status()
