"""Tensor-core path (tcgen05 projection + banded attention + ring decode) vs golden fixtures and the
CPU oracle.  Parity metric: relative L2 of the attention output <= 2e-3."""
from __future__ import annotations

import pytest
import torch

from conftest import load_golden, regen_attention_layer, regen_projections
from oracle import mimi_attention_oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-3           # attention output, relative L2
TOL_BF16_STORE = 4e-3  # q/k intermediates: one BF16 rounding of an FP32 result (not the parity metric)


def _frames(t):    # [B,H,T,D] -> [B,T,H*D]
    b, h, n, d = t.shape
    return t.transpose(1, 2).contiguous().view(b, n, h * d)


def _status_ok(st):
    import fast_mimi_b200 as fm
    assert fm.ops.read_status(st) == 0


def test_qkv_projection_rope_matches_oracle():
    import fast_mimi_b200 as fm
    torch.manual_seed(3)
    B, T = 3, 250
    x = torch.randn(B, T, 512).bfloat16()
    w = (torch.randn(1536, 512) * 0.02).bfloat16()
    cos, sin = O.rope_tables(torch.arange(T))
    q, k, v = O.qkv_project(x.float(), *w.float().chunk(3, 0))
    q, k = O.apply_rope(q, k, cos, sin)
    st = fm.ops.new_status("cuda")
    gq, gk, gv = fm.ops.qkv_rope(x.cuda(), w.cuda(), cos.cuda()[None], sin.cuda()[None], status=st)
    _status_ok(st)
    assert gv.dtype == torch.float16
    assert O.rel_l2(gq.float().cpu(), _frames(q)) < TOL_BF16_STORE
    assert O.rel_l2(gk.float().cpu(), _frames(k)) < TOL_BF16_STORE
    assert O.rel_l2(gv.float().cpu(), _frames(v)) < 5e-4


def test_qkv_projection_ragged_rows_and_per_clip_tables():
    """M = B*T not a multiple of the 128-row tile; cos/sin given per clip."""
    import fast_mimi_b200 as fm
    torch.manual_seed(4)
    B, T = 5, 37
    x = torch.randn(B, T, 512).bfloat16()
    w = (torch.randn(1536, 512) * 0.02).bfloat16()
    tabs = [O.rope_tables(torch.arange(10 * b, 10 * b + T)) for b in range(B)]
    cos = torch.stack([t[0] for t in tabs]); sin = torch.stack([t[1] for t in tabs])
    q, k, v = O.qkv_project(x.float(), *w.float().chunk(3, 0))
    q, k = O.apply_rope(q, k, cos, sin)
    gq, gk, gv = fm.ops.qkv_rope(x.cuda(), w.cuda(), cos.cuda(), sin.cuda(), value_dtype=torch.bfloat16)
    assert O.rel_l2(gq.float().cpu(), _frames(q)) < TOL_BF16_STORE
    assert O.rel_l2(gk.float().cpu(), _frames(k)) < TOL_BF16_STORE
    assert O.rel_l2(gv.float().cpu(), _frames(v)) < TOL_BF16_STORE


def test_isolated_op_config2_matches_golden():
    import fast_mimi_b200 as fm
    g = load_golden("isolated_T250.npz")
    gen = torch.Generator().manual_seed(int(g["seed"]))
    q, k, v = (torch.randn(1, 8, 250, 64, generator=gen) / 8 for _ in range(3))
    cos, sin = O.rope_tables(torch.arange(250))
    qr, kr = O.apply_rope(q, k, cos, sin)
    out = fm.native_window_attention(qr.cuda(), kr.cuda(), v.cuda(), scale=0.125, window=250)
    assert out.shape == (1, 8, 250, 64) and out.dtype == torch.float32
    assert O.rel_l2(out[0][:, g["rows"]].cpu(), g["out"]) < TOL


def test_long_band_T700_matches_golden():
    import fast_mimi_b200 as fm
    g = load_golden("band_T700.npz")
    gen = torch.Generator().manual_seed(int(g["seed"]))
    q, k, v = (torch.randn(1, 8, 700, 64, generator=gen) / 8 for _ in range(3))
    cos, sin = O.rope_tables(torch.arange(700))
    qr, kr = O.apply_rope(q, k, cos, sin)
    out = fm.native_window_attention(qr.cuda(), kr.cuda(), v.cuda(), scale=0.125, window=250)
    assert O.rel_l2(out[0][:, g["rows"]].cpu(), g["out"]) < TOL


@pytest.mark.parametrize("T", [1, 2, 63, 64, 65, 125, 127, 128, 129, 249, 250, 251, 313, 513])
@pytest.mark.parametrize("window", [250])
def test_odd_lengths_match_oracle(T, window):
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(T)
    q, k, v = (torch.randn(2, 8, T, 64, generator=gen) / 2 for _ in range(3))
    ref = O.band_attention(q, k, v, window=window, scale=0.125)
    out = fm.native_window_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.125, window=window)
    assert O.rel_l2(out.cpu(), ref) < TOL
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("window", [1, 8, 100, 128, 129, 300])
def test_other_windows_match_oracle(window):
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(window)
    q, k, v = (torch.randn(1, 8, 400, 64, generator=gen) / 2 for _ in range(3))
    ref = O.band_attention(q, k, v, window=window, scale=0.125)
    out = fm.native_window_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.125, window=window)
    assert O.rel_l2(out.cpu(), ref) < TOL


@pytest.mark.parametrize("B,T,window", [(1, 257, 250), (2, 384, 250), (1, 385, 130), (1, 640, 257), (3, 1000, 250),
                                        (20, 520, 250), (40, 300, 200), (1, 2500, 250)])
def test_long_clips_match_oracle(B, T, window):
    """Clips longer than two tiles with a window that spans three key tiles: the run-walking kernel.  The cases
    cover a ragged last tile, both window limits, runs split into segments with halo tiles (few sequences) and
    several whole-sequence runs per CTA (more sequences than SMs)."""
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(B * 10000 + T)
    q, k, v = (torch.randn(B, 8, T, 64, generator=gen) / 2 for _ in range(3))
    ref = O.band_attention_sdpa(q, k, v, window=window, scale=0.125)
    st = fm.ops.new_status("cuda")
    frames = lambda t, dt: t.transpose(1, 2).reshape(B, T, 512).to(dt).cuda()
    out = fm.ops.band_attention_prefill(frames(q, torch.bfloat16), frames(k, torch.bfloat16), frames(v, torch.float16),
                                        window=window, scale=0.125, status=st)
    _status_ok(st)
    got = out.float().cpu().view(B, T, 8, 64).transpose(1, 2)
    assert torch.isfinite(got).all()
    assert O.rel_l2(got, ref) < TOL
    # per-tile check, so that one wrong tile cannot hide in the norm of a long clip
    for t0 in range(0, T, 128):
        assert O.rel_l2(got[:, :, t0:t0 + 128], ref[:, :, t0:t0 + 128]) < TOL, t0


def test_window_attention_nlc_returns_frame_major_layout():
    """The long-sequence helper of the reference returns [1, T, 512]; ours is the same numbers as
    native_window_attention without the transpose back to [B, H, T, D]."""
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(77)
    q, k, v = (torch.randn(1, 8, 1000, 64, generator=gen) / 2 for _ in range(3))
    nlc = fm.window_attention_nlc(q.cuda(), k.cuda(), v.cuda())
    bhtd = fm.native_window_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.125, window=250)
    assert nlc.shape == (1, 1000, 512) and nlc.dtype == torch.float32
    assert torch.equal(nlc, bhtd.transpose(1, 2).reshape(1, 1000, 512))
    assert O.rel_l2(nlc.cpu().view(1, 1000, 8, 64).transpose(1, 2), O.band_attention_sdpa(q, k, v, scale=0.125)) < TOL


def test_bf16_value_path_is_available_and_close():
    """value_dtype=bfloat16 (the literal BF16 cache) is supported; its rounding alone costs ~2e-3."""
    import fast_mimi_b200 as fm
    gen = torch.Generator().manual_seed(21)
    q, k, v = (torch.randn(1, 8, 250, 64, generator=gen) / 2 for _ in range(3))
    ref = O.band_attention(q, k, v, scale=0.125)
    out = fm.native_window_attention(q.cuda(), k.cuda(), v.cuda(), scale=0.125, window=250,
                                     value_dtype=torch.bfloat16)
    assert O.rel_l2(out.cpu(), ref) < 6e-3


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("frames", [1, 127, 1000, 33 * 250])
def test_out_proj_with_layer_scale_and_residual_matches_oracle(frames, dtype):
    """o_proj with the layer scale and residual add in the epilogue; ragged frame counts, both 16-bit types,
    with and without the optional operands, and in place over the residual."""
    import fast_mimi_b200 as fm
    torch.manual_seed(11)
    a = torch.randn(frames, 512).to(dtype)
    w = (torch.randn(512, 512) * 0.05).to(dtype)
    s = torch.rand(512) * 0.5 + 0.01
    r = torch.randn(frames, 512).to(dtype)
    tol = 5e-4 if dtype == torch.float16 else 4e-3      # one rounding of the result to the output type
    st = fm.ops.new_status("cuda")
    for scale, resid in ((None, None), (s, None), (s, r)):
        ref = O.out_proj_residual(a.float(), w.float(), scale, None if resid is None else resid.float())
        got = fm.ops.out_proj(a.cuda(), w.cuda(), layer_scale=None if scale is None else scale.cuda(),
                              residual=None if resid is None else resid.cuda(), status=st)
        assert got.dtype == dtype and O.rel_l2(got.float().cpu(), ref) < tol
    buf = r.cuda().clone()
    fm.ops.out_proj(a.cuda(), w.cuda(), layer_scale=s.cuda(), residual=buf, out=buf, status=st)
    assert torch.equal(buf, got)
    _status_ok(st)


def test_out_proj_after_attention_matches_reference_layer():
    """Projection + attention + o_proj, all three on the tensor-core kernels, vs the reference layer output."""
    import fast_mimi_b200 as fm
    g = load_golden("attention_layer_T250.npz")
    x, wq, wk, wv, wo = regen_attention_layer(int(g["seed"]), int(g["b"]), int(g["t"]))
    cos, sin = O.rope_tables(torch.arange(x.shape[1]))
    core = fm.ops.attention_prefill(x.half().cuda(), torch.cat([wq, wk, wv]).half().cuda(), cos.cuda()[None],
                                    sin.cuda()[None])
    out = fm.ops.out_proj(core, wo.half().cuda())
    assert O.rel_l2(out[:, g["rows"]].float().cpu(), g["out"]) < TOL


@pytest.mark.parametrize("name", ["attention_layer_T250.npz", "attention_layer_T313.npz"])
def test_attention_module_matches_reference_layer(name):
    """MimiAttentionB200 (tensor-core path, o_proj included) vs the reference MimiAttention output."""
    import fast_mimi_b200 as fm
    g = load_golden(name)
    m = fm.MimiAttentionB200().cuda()       # constructed first: its default init consumes the RNG
    x, wq, wk, wv, wo = regen_attention_layer(int(g["seed"]), int(g["b"]), int(g["t"]))
    assert torch.equal(x[0, :2, :8], g["x_probe"])
    with torch.no_grad():
        for lin, w in zip((m.q_proj, m.k_proj, m.v_proj, m.o_proj), (wq, wk, wv, wo)):
            lin.weight.copy_(w)
    cos, sin = O.rope_tables(torch.arange(x.shape[1]))
    out, weights = m(x.cuda(), None, None, (cos.cuda()[None], sin.cuda()[None]))
    assert weights is None and out.dtype == torch.float32
    assert O.rel_l2(out[:, g["rows"]].cpu(), g["out"]) < TOL


def test_attention_module_with_full_fp32_weights_and_activations():
    """The drop-in scenario: an FP32 model whose weights and activations are NOT BF16-representable.  The
    module feeds the tensor core FP16 copies of x and W (BF16 copies alone would cost 2.4e-3)."""
    import fast_mimi_b200 as fm
    g = load_golden("attention_layer_T250_fp32.npz")
    m = fm.MimiAttentionB200().cuda()
    x, wq, wk, wv, wo = regen_attention_layer(int(g["seed"]), int(g["b"]), int(g["t"]), bf16_inputs=False)
    assert torch.equal(x[0, :2, :8], g["x_probe"]) and torch.equal(wq[:2, :8], g["wq_probe"])
    with torch.no_grad():
        for lin, w in zip((m.q_proj, m.k_proj, m.v_proj, m.o_proj), (wq, wk, wv, wo)):
            lin.weight.copy_(w)
    cos, sin = O.rope_tables(torch.arange(x.shape[1]))
    out, _ = m(x.cuda(), None, None, (cos.cuda()[None], sin.cuda()[None]))
    assert O.rel_l2(out[:, g["rows"]].cpu(), g["out"]) < TOL
    # the same module told to use BF16 inputs lands above the tolerance, which is why FP16 is the default
    m.input_dtype = torch.bfloat16
    out_bf16, _ = m(x.cuda(), None, None, (cos.cuda()[None], sin.cuda()[None]))
    assert 2e-3 < O.rel_l2(out_bf16[:, g["rows"]].cpu(), g["out"]) < 6e-3


def test_streaming_decode_260_steps_matches_reference():
    """260 one-frame steps through the KV ring (fills, then wraps at step 250) vs the reference's
    MimiKVCache + SDPA outputs; the ring must hold the same rows as the reference cache."""
    import fast_mimi_b200 as fm
    g = load_golden("ring_decode_260.npz")
    m = fm.MimiAttentionB200().cuda()
    ws = regen_projections(int(g["seed"]))
    with torch.no_grad():
        for dst, src in zip((m.q_proj, m.k_proj, m.v_proj, m.o_proj), ws):
            dst.weight.copy_(src)
    cache = m.new_cache(1, 2, "cuda")
    keep = g["keep_steps"].tolist()
    got = []
    for step in range(260):
        x = torch.randn(2, 1, 512).bfloat16().float()
        cos, sin = O.rope_tables(torch.arange(step, step + 1))
        out, _ = m(x.cuda(), None, cache, (cos.cuda()[None], sin.cuda()[None]))
        if step in keep:
            got.append(out.cpu())
    assert cache.get_seq_length() == 260
    got = torch.stack(got)
    for i, step in enumerate(keep):
        assert O.rel_l2(got[i], g["outs"][i]) < TOL, step
    k_ord, v_ord = cache.ordered(0)
    assert k_ord.shape[2] == 250
    assert O.rel_l2(k_ord[:, :, -3:].float().cpu(), g["final_key_cache"]) < TOL_BF16_STORE
    assert O.rel_l2(v_ord[:, :, -3:].float().cpu(), g["final_value_cache"]) < 5e-4


def _module_with_weights(ws):
    """``ws``: four [512, 512] weights (q, k, v, o) or a fixture seed.  The module is built BEFORE a seed's
    weights are regenerated: its own default initialisation consumes the global RNG, and the fixtures' inputs
    are drawn right after their weights."""
    import fast_mimi_b200 as fm
    m = fm.MimiAttentionB200().cuda()
    if isinstance(ws, int):
        ws = regen_projections(ws)
    with torch.no_grad():
        for dst, src in zip((m.q_proj, m.k_proj, m.v_proj, m.o_proj), ws):
            dst.weight.copy_(src)
    return m


def test_cached_multi_frame_chunks_match_reference():
    """Chunked streaming through the tensor-core path: every call carries several new frames on top of the KV
    ring (the reference's scenario of tests/test_parity.py:56-81 at Mimi's geometry: chunks that cross the
    window, one-frame steps between them, a chunk longer than the window) vs the reference's MimiAttention +
    MimiKVCache outputs; the ring must end up holding the reference cache's rows."""
    g = load_golden("cached_chunks_mimi.npz")
    m = _module_with_weights(int(g["seed"]))
    b = int(g["b"])
    cache = m.new_cache(1, b, "cuda")
    for step, t in enumerate(g["chunks"].tolist()):
        x = torch.randn(b, t, 512).bfloat16().float()
        past = cache.get_seq_length()
        cos, sin = O.rope_tables(torch.arange(past, past + t))
        out, _ = m(x.cuda(), None, cache, (cos.cuda()[None], sin.cuda()[None]))
        err = O.rel_l2(out.cpu()[:, g[f"rows{step}"]], g[f"out{step}"])
        print(f"chunk {step} (T={t}, past={past}): rel-L2 {err:.2e}")
        assert err < TOL, (step, t, err)
    assert cache.get_seq_length() == int(g["seq_length"])
    k_ord, v_ord = cache.ordered(0)
    assert O.rel_l2(k_ord[:, :, -3:].float().cpu(), g["final_key_cache"]) < TOL_BF16_STORE
    assert O.rel_l2(v_ord[:, :, -3:].float().cpu(), g["final_value_cache"]) < 5e-4
    import fast_mimi_b200 as fm
    fm.check_status()


@pytest.mark.parametrize("chunks", [[300, 1, 1], [250, 7, 1], [1, 1, 128, 129, 1], [5, 256, 257, 2]])
def test_prefill_into_ring_then_stream_equals_full_prefill(chunks):
    """Seeding the ring with a multi-frame call and continuing with chunks / single frames gives the rows of one
    cache-free prefill over the concatenated frames (the band mask makes both see the same keys)."""
    torch.manual_seed(17)
    m = _module_with_weights([torch.randn(512, 512) * 0.03 for _ in range(4)])
    total = sum(chunks)
    x = torch.randn(2, total, 512).bfloat16().float().cuda()
    cos, sin = (t.cuda()[None] for t in O.rope_tables(torch.arange(total)))
    full, _ = m(x, None, None, (cos, sin))
    cache = m.new_cache(1, 2, "cuda")
    a = 0
    for t in chunks:
        out, _ = m(x[:, a:a + t], None, cache, (cos[:, a:a + t], sin[:, a:a + t]))
        err = O.rel_l2(out.float().cpu(), full[:, a:a + t].float().cpu())
        assert err < TOL, (chunks, a, t, err)
        a += t


def test_ring_update_matches_reference_cache_semantics():
    """MimiKVRing.update (the MimiKVCache.update-compatible entry for callers that rotate K / V themselves):
    visible rows and survivors follow src/fast_mimi/model.py:450-471."""
    import fast_mimi_b200 as fm
    ring = fm.MimiKVRing(1, 2, 8, device="cuda")
    ref = O.KVCacheOracle(window=8)
    g = torch.Generator().manual_seed(3)
    for t in (3, 1, 9, 2, 1):       # values that the ring's BF16 / FP16 storage holds exactly
        k = torch.randn(2, 8, t, 64, generator=g).bfloat16().float()
        v = torch.randn(2, 8, t, 64, generator=g).half().float()
        want_k, want_v = ref.update(k, v, 0)
        got_k, got_v = ring.update(k.cuda(), v.cuda(), 0)
        assert torch.equal(got_k.cpu(), want_k) and torch.equal(got_v.cpu(), want_v), t
        assert ring.get_mask_sizes(4) == ref.get_mask_sizes(4)
    assert ring.get_seq_length() == ref.get_seq_length() == 16
    assert ring.to("cuda") is ring


def test_negative_position_is_rejected_before_any_launch():
    import fast_mimi_b200 as fm
    ring = fm.MimiKVRing(1, 2, 250, device="cuda")
    x = torch.zeros(2, 512, device="cuda", dtype=torch.bfloat16)
    w = torch.zeros(1536, 512, device="cuda", dtype=torch.bfloat16)
    cs = torch.zeros(1, 1, 64, device="cuda")
    with pytest.raises(RuntimeError):
        fm.ops.decode_step(x, w, cs, cs, ring.ring_k[0], ring.ring_v[0], -1)
    lib = fm._native.load()
    out = torch.full((2, 512), float("nan"), device="cuda")
    st = fm.ops.new_status("cuda")
    rc = lib.fm_decode_step_bf16(x.data_ptr(), w.data_ptr(), cs.data_ptr(), cs.data_ptr(), 0, None, -3, x.data_ptr(),
                                 ring.ring_k[0].data_ptr(), ring.ring_v[0].data_ptr(), out.data_ptr(), 2, 250, 0.125, 1,
                                 st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == -1
    rc = lib.fm_ring_attn_decode_bf16(x.data_ptr(), ring.ring_k[0].data_ptr(), ring.ring_v[0].data_ptr(), out.data_ptr(),
                                      None, -1, 2, 250, 0.125, 1, st.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == -1
    torch.cuda.synchronize()
    assert bool(torch.isnan(out).all()) and fm.ops.read_status(st) == 0


def test_preset_status_word_makes_kernels_return_untouched_outputs():
    """The sticky status word: a kernel handed a non-zero word must not write its outputs, and check_status must
    raise until the word is cleared."""
    import fast_mimi_b200 as fm
    st = fm.ops.new_status("cuda")
    st.fill_(101)
    x = torch.randn(2, 250, 512, device="cuda").bfloat16()
    w = (torch.randn(1536, 512, device="cuda") * 0.02).bfloat16()
    cos, sin = (t.cuda()[None] for t in O.rope_tables(torch.arange(250)))
    out = torch.full((2, 250, 512), float("nan"), device="cuda", dtype=torch.float16)
    fm.ops.attention_prefill(x, w, cos, sin, out=out, status=st)
    fm.ops.band_attention_prefill(x, x, x.half(), out=out, status=st)
    x6 = torch.randn(1, 600, 512, device="cuda").bfloat16()
    out6 = torch.full((1, 600, 512), float("nan"), device="cuda", dtype=torch.float16)
    fm.ops.band_attention_prefill(x6, x6, x6.half(), out=out6, status=st)
    fm.ops.band_attention_prefill(x6, x6, x6.half(), out=out6, window=64, status=st)
    y = torch.full((2, 250, 512), float("nan"), device="cuda", dtype=torch.float16)
    fm.ops.linear(x, w[:512].contiguous(), out=y, status=st)
    torch.cuda.synchronize()
    assert bool(torch.isnan(out.float()).all()) and bool(torch.isnan(out6.float()).all()) and bool(torch.isnan(y.float()).all())
    assert fm.ops.read_status(st) == 101
    with pytest.raises(RuntimeError, match="101"):
        fm.check_status(status=st)
    st.zero_()
    fm.check_status(status=st)
    fm.ops.attention_prefill(x, w, cos, sin, out=out, status=st)
    torch.cuda.synchronize()
    assert not bool(torch.isnan(out.float()).any())


def test_bounded_wait_gives_up_and_reports():
    """The bounded-wait machinery itself: a barrier that nothing arms, a 2 ms limit; the kernel ends by itself with
    code 103 in the status word, and a later wait in the same block returns at once."""
    import fast_mimi_b200 as fm
    lib = fm._native.load()
    st = fm.ops.new_status("cuda")
    seen = torch.full((3,), -1, dtype=torch.int32, device="cuda")
    rc = lib.fm_selftest_wait_timeout(st.data_ptr(), 2000, seen.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert fm.ops.read_status(st) == 103
    assert seen.tolist() == [0, 0, 1]
    with pytest.raises(RuntimeError, match="103"):
        fm.check_status(status=st)


@pytest.mark.parametrize("T", [129, 200, 256])
@pytest.mark.parametrize("window", [1, 8, 100, 129, 200, 256])
def test_whole_clip_kernels_with_other_windows(T, window):
    """Clips of 129..256 frames under windows that leave rows of the second tile with nothing visible in the first
    (window <= 128) and windows that cut into it: the clip-attention kernel (q, k, v given) and the fused kernel
    (x given) against the oracle."""
    import fast_mimi_b200 as fm
    torch.manual_seed(T * 1000 + window)
    x = torch.randn(2, T, 512).bfloat16()
    w = (torch.randn(1536, 512) * 0.03).bfloat16()
    cos, sin = O.rope_tables(torch.arange(T))
    q, k, v = O.qkv_project(x.float(), *w.float().chunk(3, 0))
    q, k = O.apply_rope(q, k, cos, sin)
    want = O.band_attention(q, k, v, window=window).transpose(1, 2).reshape(2, T, 512)
    dev = lambda t: t.cuda()
    fused = fm.ops.attention_fused(dev(x), dev(w), dev(cos[None]), dev(sin[None]), window=window)
    assert O.rel_l2(fused.float().cpu(), want) < TOL
    qd, kd, vd = fm.ops.qkv_rope(dev(x), dev(w), dev(cos[None]), dev(sin[None]))
    clip = fm.ops.band_attention_prefill(qd, kd, vd, window=window)
    assert O.rel_l2(clip.float().cpu(), want) < TOL
    fm.check_status()


def test_cache_free_entry_point_routes_whole_clips_to_one_kernel():
    """fm_attention_prefill_bf16: clips of 129-256 frames run as one kernel and leave the workspaces alone (null is
    accepted); other lengths need the workspaces (null is refused before any launch) and fill them."""
    import fast_mimi_b200 as fm
    from fast_mimi_b200 import _native
    lib = _native.load()
    torch.manual_seed(3)
    w = (torch.randn(1536, 512) * 0.03).bfloat16().cuda()
    stream = torch.cuda.current_stream().cuda_stream
    for T in (250, 100):
        x = torch.randn(2, T, 512).bfloat16().cuda()
        cos, sin = (t[None].contiguous().cuda() for t in O.rope_tables(torch.arange(T)))
        out = torch.zeros(2, T, 512, dtype=torch.float16, device="cuda")
        rc = lib.fm_attention_prefill_bf16(x.data_ptr(), w.data_ptr(), cos.data_ptr(), sin.data_ptr(), 0, None, None, None,
                                           out.data_ptr(), 2, T, 250, 0.125, 1, None, stream)
        torch.cuda.synchronize()
        if T > 128:
            assert rc == 0
            assert torch.equal(out, fm.ops.attention_fused(x, w, cos, sin))
            ws = [torch.full((2, T, 512), 7.0, dtype=dt, device="cuda") for dt in (torch.bfloat16, torch.bfloat16, torch.float16)]
            fm.ops.attention_prefill(x, w, cos, sin, workspace=tuple(ws))
            assert all(bool((t == 7.0).all()) for t in ws)          # untouched
        else:
            assert rc == -1 and not out.any()
            q, k, v = fm.ops.qkv_rope(x, w, cos, sin)
            want = fm.ops.band_attention_prefill(q, k, v)
            assert torch.equal(fm.ops.attention_prefill(x, w, cos, sin), want)
    fm.check_status()


@pytest.mark.parametrize("growth", [0.0, 0.05, 0.1])
def test_fused_kernel_when_later_keys_score_far_higher(growth):
    """The one-kernel form exponentiates a row against an offset taken from its first visible keys and raises it only
    when a later 32-key group exceeds it by 13 binary orders.  Frames whose magnitude grows along the clip make the
    scores of every row climb from key to key (growth 0.1: by up to about 15 binary orders per 32 keys, so the
    raise-and-rescale detour runs for most groups; 0.05: a few times per row; 0: never).  q and k are rounded to BF16
    the same way in both forms, so the check is against the two-kernel form, which subtracts the true row maximum;
    the mildest case also against the oracle."""
    import fast_mimi_b200 as fm
    torch.manual_seed(11)
    B, T = 2, 250
    u = torch.randn(512) / 8.0                                    # one direction for all frames: |u_head|^2 about 1
    amp = 1.0 + growth * torch.arange(T, dtype=torch.float32)
    x = (amp[None, :, None] * u[None, None, :] + 0.05 * torch.randn(B, T, 512)).bfloat16()
    eye = torch.eye(512)
    w = torch.cat([eye, eye, eye * 0.5 + 0.01 * torch.randn(512, 512)]).bfloat16()      # q = k = x
    cos = torch.ones(1, T, 64); sin = torch.zeros(1, T, 64)        # no rotation: q_i . k_j = a_i a_j |u_head|^2 + noise
    dev = lambda t: t.cuda()
    fused = fm.ops.attention_fused(dev(x), dev(w), dev(cos), dev(sin))
    qd, kd, vd = fm.ops.qkv_rope(dev(x), dev(w), dev(cos), dev(sin))
    two = fm.ops.band_attention_prefill(qd, kd, vd)
    fm.check_status()
    assert torch.isfinite(fused.float()).all()
    err = O.rel_l2(fused.float().cpu(), two.float().cpu())
    span = float((qd[0, -1, :64].float() * kd[0, :, :64].float()).sum(-1).max() - (qd[0, -1, :64].float() * kd[0, :, :64].float()).sum(-1).min()) * 0.125 * 1.4427
    print(f"[growth {growth}] scores of the last row span {span:.0f} binary orders; one-kernel vs two-kernel form: {err:.2e}")
    assert err < TOL
    if growth == 0.0:
        q, k, v = O.qkv_project(x.float(), *w.float().chunk(3, 0))
        want = O.band_attention(q, k, v).transpose(1, 2).reshape(B, T, 512)
        assert O.rel_l2(fused.float().cpu(), want) < TOL


# one head a pair of CTAs; two and a first pair that ends inside a clip; nine, two clips of a pair; whole clips, one and two of a pair; 17 heads; the last with
# 14 heads, the first for which whole clips are faster though some pairs get one and others two
@pytest.mark.parametrize("clips", [1, 10, 75, 74, 148, 149, 129, 131])
@pytest.mark.parametrize("T", [129, 256])
def test_heads_of_whole_clips_dealt_to_pairs_of_blocks(clips, T):
    """Which pair of blocks computes a head changes no bit: the clips, each with its own RoPE tables, in one call against
    seven at a time, and a call of one against the two-kernel form."""
    import fast_mimi_b200 as fm
    g = torch.Generator(device="cuda").manual_seed(clips + T)
    x = torch.randn(clips, T, 512, device="cuda", generator=g).bfloat16()
    w = (torch.randn(1536, 512, device="cuda", generator=g) * 0.03).bfloat16()
    cos, sin = fm.rope_tables(torch.arange(T, device="cuda") + 3 * torch.arange(clips, device="cuda")[:, None])
    out = fm.ops.attention_fused(x, w, cos, sin)
    for at in range(0, clips, 7):
        s = slice(at, at + 7)
        assert torch.equal(out[s], fm.ops.attention_fused(x[s], w, cos[s].contiguous(), sin[s].contiguous()))
    two = fm.ops.band_attention_prefill(*fm.ops.qkv_rope(x[-1:], w, cos[-1:].contiguous(), sin[-1:].contiguous()))
    assert O.rel_l2(out[-1:].float().cpu(), two.float().cpu()) < TOL
    fm.check_status()


def test_decode_with_a_different_position_per_stream_across_the_wrap():
    """16 streams at positions (37 s) % 600 + step, stepped over the ring's wrap (249 -> 250 -> 251 for some of
    them), per-stream tables [S, 1, 64] and a device-side stream_pos: every stream's step against the last row of a
    cache-free prefill over that stream's own history."""
    import fast_mimi_b200 as fm
    torch.manual_seed(5)
    S, steps = 16, 4
    w = (torch.randn(1536, 512) * 0.03).bfloat16()
    base = (torch.arange(S) * 37) % 600
    hist = [torch.randn(int(base[s]) + steps, 512).bfloat16() for s in range(S)]     # frames 0 .. base+steps-1 of stream s
    ring = fm.MimiKVRing(1, S, 250, device="cuda")
    # seed every ring with its stream's first `base` frames through the chunk path (per stream: lengths differ)
    for s in range(S):
        n = int(base[s])
        if n == 0:
            continue
        cos, sin = O.rope_tables(torch.arange(n))
        one = fm.MimiKVRing(1, 1, 250, device="cuda")
        fm.ops.attention_chunk(hist[s][None, :n].cuda(), w.cuda(), cos[None].cuda(), sin[None].cuda(), one.ring_k[0], one.ring_v[0], 0)
        ring.ring_k[0, s].copy_(one.ring_k[0, 0]); ring.ring_v[0, s].copy_(one.ring_v[0, 0])
    pos = base.to(torch.int32).cuda()
    for t in range(steps):
        xs = torch.stack([hist[s][int(base[s]) + t] for s in range(S)])
        cs = [O.rope_tables(torch.tensor([int(base[s]) + t])) for s in range(S)]
        cos = torch.stack([c[0] for c in cs]).cuda(); sin = torch.stack([c[1] for c in cs]).cuda()      # [S, 1, 64]
        got = fm.ops.decode_step(xs.cuda(), w.cuda(), cos, sin, ring.ring_k[0], ring.ring_v[0], t, stream_pos=pos).cpu()
        for s in range(S):
            n = int(base[s]) + t + 1
            c_, s_ = O.rope_tables(torch.arange(n))
            q, k, v = O.qkv_project(hist[s][None, :n].float(), *w.float().chunk(3, 0))
            q, k = O.apply_rope(q, k, c_, s_)
            want = O.band_attention(q[:, :, -1:], k, v, q_offset=n - 1).transpose(1, 2).reshape(512)
            assert O.rel_l2(got[s], want) < TOL, (s, t, n)
    fm.check_status()


def test_module_rejects_what_it_does_not_implement():
    import fast_mimi_b200 as fm
    m = fm.MimiAttentionB200().cuda()
    x = torch.zeros(1, 4, 512, device="cuda")
    cs = tuple(t.cuda()[None] for t in O.rope_tables(torch.arange(4)))
    with pytest.raises(RuntimeError):
        m(x, None, None, cs, output_attentions=True)
    with pytest.raises(RuntimeError):
        m(x, torch.ones(1, 4, device="cuda"), None, cs)            # key-padding mask
    with pytest.raises(RuntimeError):
        m(x.cpu(), None, None, cs)                                   # no CPU path
    with pytest.raises(RuntimeError):
        fm.ops.band_attention_prefill(x, x, x)                       # wrong dtype
