"""ctypes binding of ``libfast_mimi_b200.so`` (the C ABI declared in ``include/fast_mimi_b200.h``).

Mirrors how the reference binds its own native kernels (``ctypes.CDLL`` with explicit ``argtypes`` and
``restype = c_int``: src/fast_mimi/_native_cutlass.py:110-116), except that nothing is compiled at
call time and there is no fallback: a missing library raises.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import threading

import torch  # noqa: F401  (the extension module links against its libraries)

from ._build import BIND_PATH, LIB_PATH

_P, _I, _LL, _F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float

class LayerParams(ctypes.Structure):
    """``fm_layer_params`` of the header."""
    _fields_ = [("ln1_weight", _P), ("ln1_bias", _P), ("w_qkv", _P), ("w_o", _P), ("attn_scale", _P), ("ln2_weight", _P),
                ("ln2_bias", _P), ("w_fc1", _P), ("w_fc2", _P), ("mlp_scale", _P), ("ln1_eps", _F), ("ln2_eps", _F),
                ("scale", _F), ("window", _I), ("stream_dtype", _I), ("value_dtype", _I), ("ffn", _I), ("weights_settled", _I), ("vec_dtype", _I)]


class RvqStack(ctypes.Structure):
    """``fm_rvq_stack`` of the header."""
    _fields_ = [("residual", _P), ("codebooks16", _P), ("codebooks", _P), ("e_sq", _P), ("e_max", ctypes.POINTER(_F)), ("codes", _P), ("layers", _I)]


#: name -> argtypes, in header order.  tests/test_host_logic.py checks this table against the header.
SIGNATURES: dict[str, list] = {
    "fm_abi_version": [],
    "fm_layer_forward": [ctypes.POINTER(LayerParams), _P, _P, _P, _LL, _P, _P, _LL, _I, _I, _P, _P, _I, _I, _P, _P],
    "fm_qkv_rope_bf16": [_P, _P, _P, _P, _LL, _P, _P, _P, _I, _I, _I, _P, _P],
    "fm_out_proj_f16": [_P, _P, _P, _P, _P, _LL, _I, _P, _P],
    "fm_linear_f16": [_P, _P, _P, _P, _P, _LL, _I, _I, _I, _I, _I, _P, _P],
    "fm_layernorm_f16": [_P, _I, _P, _P, _F, _P, _I, _LL, _P],
    "fm_rvq_select_f32": [_P, _I, _P, _P, _P, _P, _P, _P, _LL, _I, _F, _F, _P, _P],
    "fm_conv_rows_split": [_P, _P, _P, _I, _I, _I, _I, _I, _P],
    "fm_conv_frames_split": [_P, _P, _P, _I, _I, _I, _I, _I, _P],
    "fm_linear_split_f32": [_P, _P, _LL, _I, _P, _P, _P, _LL, _I, _I, _I, _I, _I, _I, _P, _P],
    "fm_linear_split_sum_f32": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _P, _P],
    "fm_split_direct": [_LL, _I, _I],
    "fm_linear_rows_f32": [_P, _P, _P, _P, _LL, _I, _I, _I, _P, _P],
    "fm_conv_frames_f32": [_P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _P, _P],
    "fm_conv_parts_f32": [_P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _P, _P],
    "fm_upsample2_channels_f32": [_P, _P, _P, _I, _I, _I, _P],
    "fm_rvq_decode_split": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _P, _P],
    "fm_upsample2_f32": [_P, _P, _P, _I, _I, _I, _P],
    "fm_split_half": [_P, _P, _P, _LL, _P],
    "fm_rvq_encode_f32": [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, _LL, _I, _I, _F, _P, _P],
    "fm_rvq_encode_stacks_f32": [ctypes.POINTER(RvqStack), _I, _P, _P, _P, _LL, _I, _F, _P, _P],
    "fm_rvq_encode_frames_f32": [_P, _I, _P, _P, ctypes.POINTER(RvqStack), _I, _LL, _I, _F, _P, _P],
    "fm_rvq_encode_tiles_f32": [ctypes.POINTER(RvqStack), _I, _LL, _I, _F, _P, _P],
    "fm_rvq_prepare_f32": [_P, _P, _P, _LL, _F, _F, _P],
    "fm_rvq_candidates_f16": [_P, _P, _P, _P, _P, _LL, _I, _P, _P],
    "fm_rvq_select_rec_f32": [_P, _P, _P, _P, _P, _P, _P, _LL, _I, _F, _F, _P, _P],
    "fm_rvq_to_half": [_P, _P, _LL, _P],
    "fm_rvq_decode_f32": [_P, _P, _P, _LL, _I, _I, _P, _P],
    "fm_band_attn_prefill_bf16": [_P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_window_attention": [_P, _P, _P, _I, _P, _P, _P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_attention_prefill_bf16": [_P, _P, _P, _P, _LL, _P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_band_attn_chunk_bf16": [_P, _P, _P, _P, _I, _I, _I, _I, _F, _I, _P, _P],
    "fm_attention_fused_bf16": [_P, _P, _P, _P, _LL, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_attention_chunk_bf16": [_P, _P, _P, _P, _LL, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _F, _I, _P, _P],
    "fm_attention_prefill_static_bf16": [_P, _P, _P, _P, _LL, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_decode_step_bf16": [_P, _P, _P, _P, _LL, _P, _I, _P, _P, _P, _P, _I, _I, _F, _I, _P, _P],
    "fm_ring_attn_decode_bf16": [_P, _P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P],
    "fm_band_attn_fp32_verify": [_P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _F, _P, _P],
    "fm_linear_fp32_verify": [_P, _P, _P, _I, _I, _I, _P],
    "fm_rope_fp32_verify": [_P, _P, _P, _I, _I, _I, _I, _LL, _P],
    "fm_selftest_wait_timeout": [_P, _I, _P, _P],
    "fm_rvq_decode_project_f32": [_P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _P, _P, _P],
    "fm_read_status": [_P, _P],
    "fm_read_words": [_P, _P, _P, _P],
}

_lock = threading.Lock()
_lib: ctypes.CDLL | None = None


class NativeLibraryMissing(RuntimeError):
    pass


def load() -> ctypes.CDLL:
    """Load the library once.  Raises ``NativeLibraryMissing`` if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is None:
            if not os.path.exists(LIB_PATH):
                raise NativeLibraryMissing(
                    f"{LIB_PATH} is missing: build it with `python -m fast_mimi_b200._build` "
                    "(there is no CPU or PyTorch fallback for these kernels)")
            lib = ctypes.CDLL(LIB_PATH)
            for name, argtypes in SIGNATURES.items():
                fn = getattr(lib, name)
                fn.argtypes = argtypes
                fn.restype = _I
            _lib = lib
    return _lib


_bind = None


def bind():
    """The extension module with the per-call host work (``csrc/bind``), loaded once."""
    global _bind
    if _bind is None:
        load()
        with _lock:
            if _bind is None:
                if not os.path.exists(BIND_PATH):
                    raise NativeLibraryMissing(f"{BIND_PATH} is missing: build it with `python -m fast_mimi_b200._build`")
                loader = importlib.machinery.ExtensionFileLoader("_fm_bind", BIND_PATH)
                module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_fm_bind", loader))
                loader.exec_module(module)
                _bind = module
    return _bind


def check(rc: int, what: str) -> None:
    """Turn a non-zero native status into an exception, as the reference's launchers do
    (src/fast_mimi/_native_cutlass.py:163-164)."""
    if rc != 0:
        kind = {-1: "rejected geometry or a tensor without memory", -2: "grid too large", -3: "misaligned pointer",
                -4: "cuTensorMapEncodeTiled unavailable",
                -5: "more frames than the built-in workspace holds",
                -7: "workspace too small",
                -8: "no page-locked word",
                -9: "not a call for this form",
                -6: "clip length outside the fused kernel's range (128 < T <= 256)"}.get(rc, "CUDA error" if rc > 0 else "error")
        raise RuntimeError(f"{what} failed with status {rc} ({kind})")
