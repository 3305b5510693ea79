"""CPU-side tests: ABI surface, loader behaviour, ring bookkeeping, sharding (incl. 2-rank gloo)."""
from __future__ import annotations

import ctypes
import os
import re
import subprocess
import sys

import pytest
import torch

from conftest import ROOT


def _header_functions():
    text = open(os.path.join(ROOT, "include", "fast_mimi_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.findall(r"\bint\s+(fm_\w+)\s*\(([^;]*?)\)\s*;", text, flags=re.S)


def test_library_exports_every_declared_symbol():
    from fast_mimi_b200 import _build, _native
    if not os.path.exists(_build.LIB_PATH):
        _build.build()
    lib = ctypes.CDLL(_build.LIB_PATH)      # loading needs no GPU
    declared = _header_functions()
    assert len(declared) >= 10
    for name, args in declared:
        assert hasattr(lib, name), name
        assert name in _native.SIGNATURES, name
        n_args = 0 if args.strip() in ("", "void") else len(args.split(","))
        assert n_args == len(_native.SIGNATURES[name]), name
    assert set(_native.SIGNATURES) == {n for n, _ in declared}
    lib.fm_abi_version.restype = ctypes.c_int
    assert lib.fm_abi_version() == 2


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from fast_mimi_b200 import _native
    monkeypatch.setattr(_native, "_lib", None)
    monkeypatch.setattr(_native, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(_native.NativeLibraryMissing):
        _native.load()


def test_no_product_module_imports_the_oracle():
    for dirpath, _, files in os.walk(os.path.join(ROOT, "fast_mimi_b200")):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                src = open(os.path.join(dirpath, f)).read()
                assert "oracle" not in src.replace("oracle's", ""), f


def test_ring_bookkeeping_matches_reference_cache_semantics():
    """get_seq_length / get_mask_sizes must equal MimiKVCache's (src/fast_mimi/model.py:473-505), which
    the oracle restates and the golden fixtures pin."""
    from fast_mimi_b200 import MimiKVRing
    from oracle.mimi_attention_oracle import KVCacheOracle
    ring = MimiKVRing(2, 3, 8, device="cpu")
    ref = KVCacheOracle(window=8)
    for step, t in enumerate([1, 1, 3, 1, 9, 1, 1]):
        assert ring.get_mask_sizes(t) == ref.get_mask_sizes(t)
        kv = torch.zeros(3, 8, t, 64)
        ref.update(kv, kv, 0)
        ring.advance(0, t)
        assert ring.get_seq_length() == ref.get_seq_length()
    assert ring.get_seq_length(5) == 0
    with pytest.raises(ValueError):
        ring.configure_sliding_window(9)
    with pytest.raises(ValueError):
        MimiKVRing(1, 1, 257, device="cpu")


def test_ring_ordered_view_wraps():
    from fast_mimi_b200 import MimiKVRing
    ring = MimiKVRing(1, 1, 4, device="cpu")
    for pos in range(6):
        ring.ring_k[0][:, :, pos % 4] = pos
        ring.advance(0, 1)
    k, _ = ring.ordered(0)
    assert k[0, 0, :, 0].tolist() == [2, 3, 4, 5]


@pytest.mark.parametrize("change", ["pickle", "data", "copy"])
def test_a_layer_s_rings_are_the_ring(change):
    """What a layer reads and writes is the ring's own memory, also after the ring went through pickle or got new storage."""
    import copy
    import pickle
    from fast_mimi_b200 import MimiKVRing
    ring = MimiKVRing(2, 1, 4, device="cpu")
    ring.layer_rings(1)
    if change == "pickle":
        ring = pickle.loads(pickle.dumps(ring))
    elif change == "copy":
        ring = copy.deepcopy(ring)
    else:
        ring.ring_k.data, ring.ring_v.data = ring.ring_k.clone(), ring.ring_v.clone()
    for whole, part in zip((ring.ring_k, ring.ring_v), ring.layer_rings(1)):
        part[0, 3, 2] = 5.0
        assert bool((whole[1, 0, 3, 2] == 5.0).all())


def test_shard_bounds_cover_everything_once():
    from fast_mimi_b200 import shard_bounds
    for n in (0, 1, 7, 16, 512, 4096):
        for world in (1, 2, 3, 4, 8):
            spans = [shard_bounds(n, world, r) for r in range(world)]
            assert spans[0][0] == 0 and spans[-1][1] == n
            assert all(a[1] == b[0] for a, b in zip(spans, spans[1:]))
            sizes = [hi - lo for lo, hi in spans]
            assert max(sizes) - min(sizes) <= 1


_GLOO_WORKER = r"""
import os, sys, torch, torch.distributed as dist
sys.path.insert(0, os.environ["FM_ROOT"])
from fast_mimi_b200 import shard, gather_to_host
from oracle import mimi_attention_oracle as O
dist.init_process_group("gloo")
rank, world = dist.get_rank(), dist.get_world_size()
g = torch.Generator().manual_seed(0)
q, k, v = (torch.randn(5, 8, 40, 64, generator=g) for _ in range(3))   # 5 clips over 2 ranks: 3 + 2
mine = O.band_attention(shard(q, world, rank), shard(k, world, rank), shard(v, world, rank), window=16)
full = gather_to_host(mine)
if rank == 0:
    ref = O.band_attention(q, k, v, window=16)
    assert full.shape == ref.shape and torch.equal(full, ref)
    print("GLOO_OK")
dist.destroy_process_group()
"""


def test_two_rank_clip_sharding_and_host_gather_over_gloo(tmp_path):
    script = tmp_path / "worker.py"
    script.write_text(_GLOO_WORKER)
    env = dict(os.environ, FM_ROOT=ROOT, OMP_NUM_THREADS="2")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr",
           "127.0.0.1", "--master-port", "29617", str(script)]
    res = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=240)
    assert res.returncode == 0, res.stderr[-2000:]
    assert "GLOO_OK" in res.stdout


def test_layer_module_keeps_the_reference_parameter_names():
    """State-dict keys of the drop-in layer are those of the reference's MimiTransformerLayer
    (src/fast_mimi/model.py:2017-2026 with MimiAttention :1728-1747, MimiMLP :1987-1988, MimiLayerScale :1468)."""
    import fast_mimi_b200 as fm
    want = {"self_attn.q_proj.weight", "self_attn.k_proj.weight", "self_attn.v_proj.weight", "self_attn.o_proj.weight",
            "mlp.fc1.weight", "mlp.fc2.weight", "input_layernorm.weight", "input_layernorm.bias",
            "post_attention_layernorm.weight", "post_attention_layernorm.bias", "self_attn_layer_scale.scale",
            "mlp_layer_scale.scale"}
    layer = fm.MimiTransformerLayerB200()
    assert set(layer.state_dict()) == want
    import pytest
    import torch
    with pytest.raises(RuntimeError):        # no CPU path
        layer(torch.zeros(1, 4, 512), None, None, (torch.zeros(1, 4, 64), torch.zeros(1, 4, 64)), False)


def test_rope_tables_match_the_oracle():
    """fast_mimi_b200.rope_tables against the oracle's restatement (which the fixtures pin to the tables of the
    reference's MimiRotaryEmbedding), including non-zero and per-clip position offsets."""
    import torch
    import fast_mimi_b200 as fm
    from oracle import mimi_attention_oracle as O
    pos = torch.stack([torch.arange(0, 40), torch.arange(1000, 1040)])
    cos, sin = fm.rope_tables(pos)
    assert cos.shape == (2, 40, 64) and cos.dtype == torch.float32
    for b in range(2):
        oc, os_ = O.rope_tables(pos[b])
        assert torch.equal(cos[b], oc) and torch.equal(sin[b], os_)
    assert torch.equal(cos[..., :32], cos[..., 32:])


def test_kept_copies_follow_an_assigned_data():
    """A 16-bit copy of a weight is made anew when ``.data`` is assigned, also where the parameter comes back to an address it had
    (adapters merged one after the other do that) or lies in the same memory another way round, and when a module is copied."""
    import copy
    import pickle
    import numpy as np
    import fast_mimi_b200 as fm
    layer = fm.MimiTransformerLayerB200()
    reads = {"o_proj": lambda l: (l.self_attn.o_proj.weight, l.self_attn.out_weight(torch.float16)),
             "q_proj": lambda l: (l.self_attn.q_proj.weight, l.self_attn.packed_qkv_weight(torch.float16)[:512]),
             "fc1": lambda l: (l.mlp.fc1.weight, l._cast.get("fc1", l.mlp.fc1.weight, torch.float16))}
    for read in reads.values():
        w, made = read(layer)
        assert torch.equal(made, w.half()) and read(layer)[1].data_ptr() == made.data_ptr()
        memory = np.zeros(tuple(w.shape), dtype=np.float32)
        for value in (1.0, 2.0, 3.0):
            memory[:, 0] = value
            w.data = torch.from_numpy(memory)                # a storage of its own at the same address
            assert torch.equal(read(layer)[1], w.half()), value
            if w.shape[0] == w.shape[1]:
                w.data = w.data.t()
                assert torch.equal(read(layer)[1], w.half()), value
    for other in (copy.deepcopy(layer), pickle.loads(pickle.dumps(layer))):
        with torch.no_grad():
            for w in (other.self_attn.o_proj.weight, other.self_attn.q_proj.weight, other.mlp.fc1.weight):
                w.data = w.data + 1.0
        for read in reads.values():
            assert torch.equal(read(other)[1], read(other)[0].half())


@pytest.mark.skipif(torch.cuda.is_available(), reason="made-up addresses: only where nothing can be launched")
@pytest.mark.parametrize("offset", [4, 8])
@pytest.mark.parametrize("rows", [1, 40, 5000])
def test_misaligned_rotary_tables_are_refused(rows, offset):
    """The projections read the tables 16 bytes at a time: a table that starts between such addresses is an error of the call
    (-3) on every path, before anything is launched.  The addresses are made up; nothing looks behind them."""
    import ctypes
    from fast_mimi_b200 import _native
    lib = _native.load()
    a, n = 1 << 20, None
    params = _native.LayerParams(*[a] * 10, 1e-5, 1e-5, 0.125, 250, 2, 1, 2048, 0, 2)
    for cos, sin in ((a + offset, a), (a, a + offset)):
        assert lib.fm_qkv_rope_bf16(a, a, cos, sin, 0, a, a, a, 1, rows, 1, n, n) == -3
        assert lib.fm_layer_forward(ctypes.byref(params), a, a, a, 1 << 40, cos, sin, 0, 1, rows, n, n, 0, 0, n, n) == -3
        assert lib.fm_attention_prefill_bf16(a, a, cos, sin, 0, a, a, a, a, 1, rows, 250, 0.125, 1, n, n) == -3
        assert lib.fm_attention_chunk_bf16(a, a, cos, sin, 0, a, a, a, a, a, a, a, a, 1, rows, 300, 250, 250, 0.125, 1, n, n) == -3
        assert lib.fm_decode_step_bf16(a, a, cos, sin, 0, n, 300, a, a, a, a, 1, 250, 0.125, 1, n, n) == -3


# Entry points and arguments of an ordinary call: P a tensor that has to be there, O one that a kernel behind the first needs or that may be left out.
P, O, N = "P", "O", None
CALLS = {
    "fm_qkv_rope_bf16": [P, P, P, P, 0, O, O, O, 2, 100, 0, N, N],
    "fm_out_proj_f16": [P, P, N, N, P, 64, 1, N, N],
    "fm_linear_f16": [P, P, N, N, P, 64, 512, 512, 1, 2, 0, N, N],
    "fm_layernorm_f16": [P, 2, P, P, 1e-5, P, 1, 64, N],
    "fm_rvq_select_f32": [P, 2, P, P, P, P, P, N, 64, 2048, 1.0, 1e-3, N, N],
    "fm_conv_rows_split": [P, P, P, 2, 50, 512, 4, 2, N],
    "fm_conv_frames_split": [P, P, P, 2, 50, 512, 4, 2, N],
    "fm_linear_split_f32": [P, P, 64, 512, P, P, P, 64, 1, 1, 0, 1, 512, 512, N, N],
    "fm_linear_split_sum_f32": [P, P, P, P, P, 2, 50, 512, 512, N, N],
    "fm_linear_rows_f32": [P, P, P, P, 64, 1, 512, 512, N, N],
    "fm_conv_frames_f32": [P, P, P, P, 2, 50, 512, 4, 2, 512, N, N],
    "fm_conv_parts_f32": [P, P, P, O, O, O, 2, 50, 512, 4, 2, 512, N, N],
    "fm_upsample2_channels_f32": [P, P, P, 2, 50, 512, N],
    "fm_upsample2_f32": [P, P, P, 2, 50, 512, N],
    "fm_rvq_decode_split": [P, P, P, P, P, 2, 50, 8, 1, 2048, 2048, N, N],
    "fm_split_half": [P, P, P, 64, N],
    "fm_rvq_prepare_f32": [P, P, P, 64, 1.0, 1e-3, N],
    "fm_rvq_candidates_f16": [P, P, P, P, P, 64, 2048, N, N],
    "fm_rvq_select_rec_f32": [P, P, P, P, P, N, P, 64, 2048, 1.0, 1e-3, N, N],
    "fm_rvq_to_half": [P, P, 64, N],
    "fm_rvq_decode_f32": [P, P, P, 64, 8, 2048, N, N],
    "fm_band_attn_prefill_bf16": [P, P, P, P, 2, 100, 250, 0.125, 1, N, N],
    "fm_attention_prefill_bf16": [P, P, P, P, 0, P, P, P, O, 2, 100, 250, 0.125, 1, N, N],
    "fm_band_attn_chunk_bf16": [P, P, P, P, 2, 50, 100, 250, 0.125, 1, N, N],
    "fm_attention_fused_bf16": [P, P, P, P, 0, P, 2, 200, 250, 0.125, 1, N, N],
    "fm_attention_chunk_bf16": [P, P, P, P, 0, P, P, P, O, O, P, P, P, 2, 50, 100, 250, 250, 0.125, 1, N, N],
    "fm_decode_step_bf16": [P, P, P, P, 0, N, 5, P, P, P, O, 2, 250, 0.125, 1, N, N],
    "fm_ring_attn_decode_bf16": [P, P, P, P, N, 5, 2, 250, 0.125, 1, N, N],
    "fm_band_attn_fp32_verify": [P, P, P, P, 2, 8, 64, 50, 50, 0, 0, 250, 0.125, O, N],
    "fm_linear_fp32_verify": [P, P, P, 4, 4, 4, N],
    "fm_rope_fp32_verify": [P, P, P, 1, 4, 8, 64, 0, N],
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are the host's")
def test_a_tensor_without_memory_is_refused_on_the_host():
    """A null address where a call needs a tensor (what torch's fake tensors, which say that they lie on the device, give for theirs) is an argument that
    the call rejects before it launches anything: -1, where a launch on this machine would be a CUDA error."""
    from fast_mimi_b200 import _native
    lib = _native.load()
    memory = ctypes.create_string_buffer(1 << 16)
    at = (ctypes.addressof(memory) + 1023) & ~1023
    fill = lambda a: at if a in (P, O) else a
    for name, args in CALLS.items():
        assert len(args) == len(_native.SIGNATURES[name]), name
        for i, a in enumerate(args):
            if a is P:
                assert getattr(lib, name)(*[None if j == i else fill(b) for j, b in enumerate(args)]) == -1, (name, i)
    pointers = [n for n, t in _native.LayerParams._fields_ if t is ctypes.c_void_p]
    params = lambda without: ctypes.byref(_native.LayerParams(*[None if n == without else at for n in pointers], 1e-5, 1e-5, 0.125, 250, 2, 3, 2048, 0, 2))
    call = lambda p, x, y, cos, sin: lib.fm_layer_forward(p, x, y, at, 1 << 30, cos, sin, 0, 1, 20, None, None, 0, 0, None, None)
    for n in pointers:
        if not n.endswith("scale"):
            assert call(params(n), at, at, at, at) == -1, n
    for i in range(4):
        assert call(params(None), *[None if i == j else at for j in range(4)]) == -1, i
