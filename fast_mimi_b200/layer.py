"""Drop-in replacement for the reference's transformer layer on B200.

``MimiTransformerLayerB200.forward`` keeps the signature and return type of the reference's
``MimiTransformerLayer.forward`` (src/fast_mimi/model.py:2026-2061) and its sub-module names
(``self_attn``, ``mlp.fc1``, ``mlp.fc2``, ``input_layernorm``, ``post_attention_layernorm``,
``self_attn_layer_scale.scale``, ``mlp_layer_scale.scale``), so state dicts are interchangeable.

The whole layer runs on this package's kernels, behind one native call (``ops.layer_forward``) that issues them as a
chain of dependent launches:

    LayerNorm -> QKV projection + RoPE + banded attention -> o_proj + layer scale + residual
              -> LayerNorm -> fc1 + GELU -> fc2 + layer scale + residual

The residual stream keeps the caller's dtype (FP32 stays FP32: both residual adds happen in the FP32 epilogue
of a GEMM); only the operands of the tensor-core products are rounded to 16 bit.  Calls with a cache (a
``MimiKVRing``) differ only in the attention core: up to eight new frames per stream read and update the ring in one
kernel, longer chunks of few streams take the kernel for few query tiles (which reads the ring where it lies), all others
lay ring and new rows out frame by frame for the tiled kernel.  A ring whose values have not the module's type, or a cache
of another kind, takes the attention module's kernels one by one.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _native, ops
from ._origin import Origin
from .attention import MimiAttentionB200
from .kv_ring import MimiKVRing


class _LayerScale(nn.Module):
    """Per-channel factor, as the reference's ``MimiLayerScale`` (src/fast_mimi/model.py:1454-1480)."""

    def __init__(self, channels: int, initial: float = 0.01) -> None:
        super().__init__()
        self.scale = nn.Parameter(torch.full((channels,), initial))

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return self.scale * x


class _MLP(nn.Module):
    """``fc2(gelu(fc1(x)))`` with bias-free linears (src/fast_mimi/model.py:1987-1999)."""

    def __init__(self, hidden: int, intermediate: int) -> None:
        super().__init__()
        self.fc1 = nn.Linear(hidden, intermediate, bias=False)
        self.fc2 = nn.Linear(intermediate, hidden, bias=False)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return self.fc2(F.gelu(self.fc1(x)))


class _Cast16:
    """16-bit copies of parameters, rebuilt when the parameter (or the requested type) changes."""

    def __init__(self) -> None:
        self._store: dict = {}

    def __setstate__(self, state) -> None:
        self._store = {}                        # a copied or unpickled module makes its own

    def get(self, name: str, p: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
        hit = self._store.get(name)
        if hit is None or hit[1].dtype != dtype or not hit[0].still(p):
            hit = (Origin(p), p.detach().to(dtype).contiguous())
            self._store[name] = hit
        return hit[1]


class MimiTransformerLayerB200(nn.Module):
    _plan = None            # of the class, so that layers pickled before there were plans have none

    def __init__(self, hidden_size: int = 512, intermediate_size: int = 2048, num_heads: int = 8, head_dim: int = 64,
                 sliding_window: int = 250, layer_idx: int = 0, norm_eps: float = 1e-5,
                 layer_scale_initial_scale: float = 0.01, value_dtype: torch.dtype = torch.float16) -> None:
        super().__init__()
        self.self_attn = MimiAttentionB200(hidden_size, num_heads, head_dim, sliding_window, layer_idx, "tc", value_dtype)
        self.mlp = _MLP(hidden_size, intermediate_size)
        self.input_layernorm = nn.LayerNorm(hidden_size, eps=norm_eps)
        self.post_attention_layernorm = nn.LayerNorm(hidden_size, eps=norm_eps)
        self.self_attn_layer_scale = _LayerScale(hidden_size, layer_scale_initial_scale)
        self.mlp_layer_scale = _LayerScale(hidden_size, layer_scale_initial_scale)
        self._cast = _Cast16()

    @classmethod
    def from_reference(cls, layer: nn.Module, value_dtype: torch.dtype = torch.float16) -> "MimiTransformerLayerB200":
        """Build from a module with the reference layer's attributes; every parameter is shared, not copied."""
        attn = layer.self_attn
        new = cls(attn.q_proj.in_features, layer.mlp.fc1.out_features, attn.num_heads, attn.head_dim,
                  attn.sliding_window, attn.layer_idx, layer.input_layernorm.eps, value_dtype=value_dtype)
        new.self_attn = attn if isinstance(attn, MimiAttentionB200) else MimiAttentionB200.from_reference(
            attn, "tc", value_dtype)
        new.mlp = layer.mlp
        new.input_layernorm = layer.input_layernorm
        new.post_attention_layernorm = layer.post_attention_layernorm
        new.self_attn_layer_scale = layer.self_attn_layer_scale
        new.mlp_layer_scale = layer.mlp_layer_scale
        return new

    def __getstate__(self) -> dict:
        return {**self.__dict__, "_plan": None}         # device addresses: rebuilt by the copy's first call

    def _native_plan(self, x: torch.Tensor):
        """The parameter block of the native call for activations like ``x`` (16-bit weights, LayerNorm parameters and
        layer scales) and, where every parameter is an entry of its module, the plan that notices when one of them, a
        submodule or an option changes."""
        attn, mlp, ln1, ln2 = self.self_attn, self.mlp, self.input_layernorm, self.post_attention_layernorm
        ops._need(x.dtype in ops._OUT_CODES, "x must be bfloat16, float16 or float32")
        if mlp.fc1.bias is not None or attn.o_proj.bias is not None:
            raise RuntimeError("the fused layer expects bias-free projections, as in Mimi's checkpoints")
        fc1, fc2 = mlp.fc1.weight, mlp.fc2.weight
        ffn = fc1.shape[0]
        ops._need(tuple(fc1.shape) == (ffn, 512) and tuple(fc2.shape) == (512, ffn) and ffn % 256 == 0,
                  "the MLP must be 512 -> n -> 512 with n a multiple of 256")
        tc = attn._tc_input_dtype(x)
        vectors = (ln1.weight, ln1.bias, self.self_attn_layer_scale.scale, ln2.weight, ln2.bias, self.mlp_layer_scale.scale)
        # Read where they lie if they have one type (FP32 in an FP32 residual stream); else as FP32 copies made for this call alone (no plan), since a write
        # through ``.data`` would not show in a kept copy.
        in_place = (len({p.dtype for p in vectors}) == 1 and vectors[0].dtype in ops._OUT_CODES
                    and (x.dtype != torch.float32 or vectors[0].dtype == torch.float32)
                    and all(p.is_contiguous() and p.data_ptr() % 16 == 0 for p in vectors))
        w1, b1, s1, w2, b2, s2 = (p.detach() if in_place else p.detach().float().contiguous() for p in vectors)
        keep = (w1, b1, attn.packed_qkv_weight(tc), attn.out_weight(attn.value_dtype), s1, w2, b2, self._cast.get("fc1", fc1, tc),
                self._cast.get("fc2", fc2, tc), s2)
        for t in keep:
            ops._need(t.is_cuda, "the layer's parameters must be on a CUDA device")
        params = _native.LayerParams(*(t.data_ptr() for t in keep), ln1.eps, ln2.eps, attn.scaling, attn.sliding_window,
                                     ops._OUT_CODES[x.dtype],
                                     ops._VALUE_CODES[attn.value_dtype] | (2 if tc == torch.float16 else 0), ffn, 0, ops._OUT_CODES[w1.dtype])
        self._plan = None
        if not in_place:
            return params, keep
        watches = [(self._modules, n) for n in ("self_attn", "mlp", "input_layernorm", "post_attention_layernorm",
                                                "self_attn_layer_scale", "mlp_layer_scale")]
        watches += [(attn._modules, n) for n in ("q_proj", "k_proj", "v_proj", "o_proj")]
        watches += [(mlp._modules, "fc1"), (mlp._modules, "fc2")]
        watches += [(m._parameters, "weight") for m in (ln1, ln2, attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj, mlp.fc1, mlp.fc2)]
        watches += [(m._parameters, "bias") for m in (ln1, ln2, attn.o_proj, mlp.fc1)]
        watches += [(m._parameters, "scale") for m in (self.self_attn_layer_scale, self.mlp_layer_scale)]
        watches += [(attn.__dict__, n) for n in ("sliding_window", "scaling", "value_dtype", "input_dtype")]
        watches += [(ln1.__dict__, "eps"), (ln2.__dict__, "eps")]
        try:
            like_value = torch.empty(0, dtype=attn.value_dtype)
            self._plan = _native.bind().LayerPlan(watches, keep, ctypes.addressof(params), ops.default_status(x.device), x, like_value)
        except KeyError:            # a computed parameter (parametrised weights and the like): nothing to watch
            pass
        return params, keep

    def _forward_checked(self, x, cos, sin, cache, past) -> torch.Tensor:
        """The call with everything looked at: arguments of other types or layouts, changed parameters, errors."""
        attn = self.self_attn
        x = x.contiguous()
        cos, sin = cos.to(torch.float32).contiguous(), sin.to(torch.float32).contiguous()
        params, keep = self._native_plan(x)
        if self._plan is not None:
            y = _native.bind().layer_forward(self._plan, x, cos, sin, *self._rings(cache), past)
            if isinstance(y, torch.Tensor):
                return y
        return ops.layer_forward(params, x, cos, sin, value_dtype=attn.value_dtype,
                                 ring=None if cache is None else cache.layer_rings(attn.layer_idx), past=past,
                                 window=attn.sliding_window)

    def _rings(self, cache) -> tuple:
        """What the native call takes of a cache: the rings of all layers and the layer's number in them."""
        return (None, None, 0) if cache is None else (cache.ring_k, cache.ring_v, self.self_attn.layer_idx)

    def forward(self, hidden_states: torch.Tensor, attention_mask: torch.Tensor | None, past_key_values,
                position_embeddings: tuple[torch.Tensor, torch.Tensor], output_attentions: bool = False,
                canonical_window_mask: bool = False) -> tuple[torch.Tensor, torch.Tensor | None]:
        if output_attentions:
            raise RuntimeError("attention probabilities are not materialised by the B200 kernels")
        if not hidden_states.is_cuda:
            raise RuntimeError("MimiTransformerLayerB200 runs on a CUDA device only; there is no CPU path")
        if attention_mask is not None and attention_mask.dim() != 4:
            raise RuntimeError("key-padding masks are not supported; pass None or the 4-D causal band mask")
        cache = past_key_values
        if cache is None or isinstance(cache, MimiKVRing):
            past = 0
            if cache is not None:
                attn = self.self_attn
                ops._need(cache.num_streams == hidden_states.shape[0], "cache was created for a different number of streams")
                ops._need(cache.sliding_window == attn.sliding_window, "cache window differs from the module's")
                past = cache.get_seq_length(attn.layer_idx)
            cos, sin = position_embeddings
            out = None
            if self._plan is not None:
                out = _native.bind().layer_forward(self._plan, hidden_states, cos, sin, *self._rings(cache), past)
            if type(out) is int:
                _native.check(out, "fm_layer_forward")
            if out is None and (cache is None or cache.ring_v.dtype == self.self_attn.value_dtype):
                out = self._forward_checked(hidden_states, cos, sin, cache, past)
            if out is not None:
                if cache is not None:
                    cache.advance(attn.layer_idx, hidden_states.shape[1])
                return out, None
        if self.mlp.fc1.bias is not None or self.self_attn.o_proj.bias is not None:
            raise RuntimeError("the fused layer expects bias-free projections, as in Mimi's checkpoints")
        attn = self.self_attn
        x = hidden_states.contiguous()
        # a cache object of another kind, or a ring whose values have not the module's type: the kernels one by one around the
        # attention's own way with it
        stream_dtype = x.dtype
        tc = attn._tc_input_dtype(x)
        cos, sin = (t.to(torch.float32).contiguous() for t in position_embeddings)
        ln1, ln2 = self.input_layernorm, self.post_attention_layernorm
        f32 = lambda p: p.detach().float().contiguous()       # no copy for FP32 parameters
        h = ops.layer_norm(x, f32(ln1.weight), f32(ln1.bias), eps=ln1.eps, out_dtype=tc)
        core = attn._forward_tc(h, past_key_values, cos, sin)      # FP32 from the one-frame kernel, else the ring's type
        if core.dtype not in ops._VALUE_CODES:
            core = core.to(attn.value_dtype)
        x1 = ops.linear(core, attn.out_weight(core.dtype), scale=f32(self.self_attn_layer_scale.scale), residual=x,
                        out_dtype=stream_dtype)
        h2 = ops.layer_norm(x1, f32(ln2.weight), f32(ln2.bias), eps=ln2.eps, out_dtype=tc)
        g = ops.linear(h2, self._cast.get("fc1", self.mlp.fc1.weight, tc), activation="gelu", out_dtype=tc)
        x2 = ops.linear(g, self._cast.get("fc2", self.mlp.fc2.weight, tc), scale=f32(self.mlp_layer_scale.scale),
                        residual=x1, out_dtype=stream_dtype)
        return x2, None


def install_layers(transformer: nn.Module, value_dtype: torch.dtype = torch.float16) -> nn.Module:
    """Replace every layer of a reference ``MimiTransformerModel`` (its ``layers`` ModuleList,
    src/fast_mimi/model.py:2064-2232) by a ``MimiTransformerLayerB200`` that shares its parameters."""
    for i, layer in enumerate(transformer.layers):
        transformer.layers[i] = MimiTransformerLayerB200.from_reference(layer, value_dtype)
    return transformer
