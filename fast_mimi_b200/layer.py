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
``MimiKVRing``) differ only in the attention core: ring decode for one new frame per stream, the chunk path for
several; LayerNorms, projections and the MLP are the same kernels.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _native, ops
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

    def get(self, name: str, p: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
        key = (p.data_ptr(), p._version, p.device, dtype)
        hit = self._store.get(name)
        if hit is None or hit[0] != key:
            hit = (key, p.detach().to(dtype).contiguous())
            self._store[name] = hit
        return hit[1]


class _LayerPlan:
    """What one native layer call needs besides its activations: the 16-bit weights, FP32 LayerNorm parameters and layer
    scales, and the struct that points at them."""

    def __init__(self, layer: "MimiTransformerLayerB200", x: torch.Tensor, ps: tuple, key: list) -> None:
        attn = layer.self_attn
        ops._need(x.dtype in ops._OUT_CODES, "x must be bfloat16, float16 or float32")
        ffn = ps[9].shape[0]
        ops._need(tuple(ps[9].shape) == (ffn, 512) and tuple(ps[10].shape) == (512, ffn) and ffn % 256 == 0,
                  "the MLP must be 512 -> n -> 512 with n a multiple of 256")
        tc = attn._tc_input_dtype(x)
        f32 = lambda p: p.detach().float().contiguous()       # no copy for FP32 parameters
        self.key = key
        self.keep = (f32(ps[0]), f32(ps[1]), attn.packed_qkv_weight(tc), attn.out_weight(attn.value_dtype), f32(ps[6]),
                     f32(ps[7]), f32(ps[8]), layer._cast.get("fc1", ps[9], tc), layer._cast.get("fc2", ps[10], tc), f32(ps[11]))
        for t in self.keep:
            ops._need(t.is_cuda, "the layer's parameters must be on a CUDA device")
        self.params = _native.LayerParams(*(t.data_ptr() for t in self.keep), layer.input_layernorm.eps,
                                          layer.post_attention_layernorm.eps, attn.scaling, attn.sliding_window,
                                          ops._OUT_CODES[x.dtype],
                                          ops._VALUE_CODES[attn.value_dtype] | (2 if tc == torch.float16 else 0), ffn)


class MimiTransformerLayerB200(nn.Module):
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
        self._plan: _LayerPlan | None = None

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

    def _parameters_in_use(self) -> tuple:
        """The layer's parameters, looked up in the modules' own tables (an attribute access per level costs more host
        time than a launch)."""
        m = self._modules
        try:
            a, mlp = m["self_attn"]._modules, m["mlp"]._modules
            ln1, ln2 = m["input_layernorm"]._parameters, m["post_attention_layernorm"]._parameters
            return (ln1["weight"], ln1["bias"], a["q_proj"]._parameters["weight"], a["k_proj"]._parameters["weight"],
                    a["v_proj"]._parameters["weight"], a["o_proj"]._parameters["weight"],
                    m["self_attn_layer_scale"]._parameters["scale"], ln2["weight"], ln2["bias"],
                    mlp["fc1"]._parameters["weight"], mlp["fc2"]._parameters["weight"], m["mlp_layer_scale"]._parameters["scale"])
        except KeyError:         # a parameter that is computed (parametrised weights and the like)
            at, ln1, ln2 = self.self_attn, self.input_layernorm, self.post_attention_layernorm
            return (ln1.weight, ln1.bias, at.q_proj.weight, at.k_proj.weight, at.v_proj.weight, at.o_proj.weight,
                    self.self_attn_layer_scale.scale, ln2.weight, ln2.bias, self.mlp.fc1.weight, self.mlp.fc2.weight,
                    self.mlp_layer_scale.scale)

    def _native_plan(self, x: torch.Tensor) -> "_LayerPlan":
        """The parameter block of the native call for activations like ``x``; rebuilt when a parameter was replaced or
        written to, or when an option it depends on changed."""
        attn = self.self_attn
        ps = self._parameters_in_use()
        key = [x.dtype, x.device, attn.sliding_window, attn.scaling, attn.value_dtype, attn.input_dtype,
               self.input_layernorm.eps, self.post_attention_layernorm.eps]
        for p in ps:
            key.append(p.data_ptr())
            key.append(p._version)
        plan = self._plan
        if plan is None or plan.key != key:
            plan = self._plan = _LayerPlan(self, x, ps, key)
        return plan

    def forward(self, hidden_states: torch.Tensor, attention_mask: torch.Tensor | None, past_key_values,
                position_embeddings: tuple[torch.Tensor, torch.Tensor], output_attentions: bool = False,
                canonical_window_mask: bool = False) -> tuple[torch.Tensor, torch.Tensor | None]:
        if output_attentions:
            raise RuntimeError("attention probabilities are not materialised by the B200 kernels")
        if not hidden_states.is_cuda:
            raise RuntimeError("MimiTransformerLayerB200 runs on a CUDA device only; there is no CPU path")
        if attention_mask is not None and attention_mask.dim() != 4:
            raise RuntimeError("key-padding masks are not supported; pass None or the 4-D causal band mask")
        if self.mlp.fc1.bias is not None or self.self_attn.o_proj.bias is not None:
            raise RuntimeError("the fused layer expects bias-free projections, as in Mimi's checkpoints")
        attn = self.self_attn
        x = hidden_states.contiguous()
        cache = past_key_values
        if cache is None or isinstance(cache, MimiKVRing):
            cos, sin = position_embeddings
            if cos.dtype != torch.float32 or sin.dtype != torch.float32:
                cos, sin = cos.to(torch.float32), sin.to(torch.float32)
            plan = self._native_plan(x)
            window, ring, past = attn.sliding_window, None, 0
            if cache is not None:
                ops._need(cache.num_streams == x.shape[0], "cache was created for a different number of streams")
                ops._need(cache.sliding_window == window, "cache window differs from the module's")
                ring, past = cache.layer_rings(attn.layer_idx), cache.get_seq_length(attn.layer_idx)
            out = ops.layer_forward(plan.params, x, cos.contiguous(), sin.contiguous(), value_dtype=attn.value_dtype, ring=ring,
                                    past=past, window=window)
            if cache is not None:
                cache.advance(attn.layer_idx, x.shape[1])
            return out, None
        # a cache object of another kind: the kernels one by one around its own update
        stream_dtype = x.dtype
        tc = attn._tc_input_dtype(x)
        cos, sin = (t.to(torch.float32).contiguous() for t in position_embeddings)
        ln1, ln2 = self.input_layernorm, self.post_attention_layernorm
        f32 = lambda p: p.detach().float().contiguous()       # no copy for FP32 parameters
        h = ops.layer_norm(x, f32(ln1.weight), f32(ln1.bias), eps=ln1.eps, out_dtype=tc)
        core = attn._forward_tc(h, past_key_values, cos, sin)
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
