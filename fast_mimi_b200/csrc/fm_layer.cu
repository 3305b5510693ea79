// One transformer layer behind one entry point (sm_100a): the launches of
//
//   LayerNorm -> QKV projection + RoPE -> attention -> o_proj + scale + residual
//             -> LayerNorm -> fc1 + GELU -> fc2 + scale + residual
//
// as a chain of dependent launches (reference: MimiTransformerLayer.forward, src/fast_mimi/model.py:2026-2061).
//
// For few rows a layer is bound by what surrounds the arithmetic: driven kernel by kernel from Python a layer of one
// clip cost 165 us of host time (checks, allocations, tensor maps, launches) for 84 us of GPU time.  Here the host makes
// one call; the intermediate tensors live in one workspace of the caller; and every launch but those of other libraries
// is allowed to begin (barriers, tensor memory, weight loads) while the kernel in front still runs.  Up to 168 rows everything
// behind the attention is one kernel (fm_layer_tail.cu).
#include "../../include/fast_mimi_b200.h"

#include "fm_kernels.h"

namespace fm {

namespace {
struct Arena {
  uint8_t* base;
  long long used;
  uint8_t* take(long long bytes) {
    uint8_t* p = base == nullptr ? nullptr : base + used;
    used += (bytes + 255) & ~255ll;
    return p;
  }
};

struct Buffers {
  void *h, *q, *k, *v, *core, *x1, *g, *k_lin, *v_lin;
};

// The workspace of one call.  `lin_rows`: cached and new rows laid out frame by frame (the linearised path only).
long long lay_out(uint8_t* base, long long rows, int elem, int ffn, long long lin_rows, Buffers* b) {
  Arena a = {base, 0};
  b->h = a.take(rows * 1024);
  b->core = a.take(rows * 1024);
  b->x1 = a.take(rows * 512 * elem);
  // q, k, v and the linearised ring are dead before fc1 writes g
  const long long mark = a.used;
  b->q = a.take(rows * 1024);
  b->k = a.take(rows * 1024);
  b->v = a.take(rows * 1024);
  b->k_lin = a.take(lin_rows * 1024);
  b->v_lin = a.take(lin_rows * 1024);
  const long long attn_end = a.used;
  a.used = mark;
  b->g = a.take(rows * ffn * 2);
  return a.used > attn_end ? a.used : attn_end;
}
}  // namespace

static int layer_forward(const fm_layer_params& p, const void* x, void* y, void* workspace, long long workspace_bytes,
                         const float* cos, const float* sin, long long cos_bstride, int B, int T, void* ring_k,
                         void* ring_v, int past, int slots, int* status, cudaStream_t st) {
  const long long rows_ll = static_cast<long long>(B) * T;
  if (B < 0 || T < 0 || rows_ll > 0x7fffffffLL || p.window <= 0 || p.ffn <= 0 || p.ffn % 256 != 0) return -1;
  if (rows_ll == 0) return 0;
  if (absent(x, y, cos, sin) || absent(p.ln1_weight, p.ln1_bias, p.w_qkv, p.w_o, p.ln2_weight, p.ln2_bias, p.w_fc1, p.w_fc2)) return -1;
  if (!rope_tables_aligned(cos, sin, cos_bstride)) return -3;
  const bool cached = ring_k != nullptr;
  if (cached && (ring_v == nullptr || past < 0 || slots < p.window)) return -1;
  const int rows = static_cast<int>(rows_ll);
  const int delta = cached ? (past < p.window - 1 ? past : p.window - 1) : 0;
  const bool few = cached && slots <= 256 && T <= 8;           // fm_stream_attn.cu
  const bool whole_clip = !cached && T > 128 && T <= 256;
  const long long lin_rows = cached && !few && delta > 0 ? static_cast<long long>(B) * (delta + T) : 0;
  Buffers b;
  if (lay_out(static_cast<uint8_t*>(workspace), rows, p.stream_dtype == 2 ? 4 : 2, p.ffn, lin_rows, &b) > workspace_bytes) return -7;
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) return -3;
  const auto vec = [&](const void* v) { return ParamVec(v, p.vec_dtype); };
  const int value_fp16 = p.value_dtype & 1;
  const int tc = (p.value_dtype & 2) ? 1 : 0;                    // 16-bit type of the products' operands: 0 BF16, 1 FP16

  const bool front = few && stream_front_takes(B, T, slots);    // everything up to the attention is one kernel
  const bool norm1_inside = few_rows_with_norm(rows, 1536), norm2_inside = few_rows_with_norm(rows, p.ffn);
  int rc = 0;
  if (!norm1_inside && !front) {
    rc = launch_layernorm512(x, p.stream_dtype, vec(p.ln1_weight), vec(p.ln1_bias), p.ln1_eps, b.h, tc, rows, st, 1);
    if (rc != 0) return rc;
  }
  const bool one_tail = layer_tail_takes(rows, p.ffn);          // everything behind the attention is one kernel
  const bool few_tiles = !few && few_attn_tiles(B, T) && (!cached || slots <= 256);
  if (front) {
    const StreamFront f = {x, vec(p.ln1_weight), vec(p.ln1_bias), p.ln1_eps, p.w_qkv, cos, sin, cos_bstride, ring_k, ring_v, b.core, p.stream_dtype,
                           value_fp16, tc};
    rc = launch_stream_front(f, B, T, past, slots, p.window, p.scale, status, st, p.weights_settled);
  } else if (whole_clip && !few_tiles && use_fused_clip(B, T)) {
    rc = launch_attn_fused_clip(b.h, p.w_qkv, cos, sin, cos_bstride, b.core, B, T, p.window, p.scale, p.value_dtype, status, st, 1);
  } else {
    QkvEpilogueArgs ep = {};
    ep.q = static_cast<uint16_t*>(b.q);
    ep.k = static_cast<uint16_t*>(b.k);
    ep.v = static_cast<uint16_t*>(b.v);
    ep.cos = cos;
    ep.sin = sin;
    ep.cos_bstride = cos_bstride;
    ep.T = T;
    ep.ring_slots = 1;
    // The kernel that opens the chain may ask for W_qkv ahead of its wait only if W_qkv cannot be the work of the kernel
    // in front: not on the first call after the caller has (re)made it.
    rc = norm1_inside ? launch_ln_qkv(x, p.stream_dtype, vec(p.ln1_weight), vec(p.ln1_bias), p.ln1_eps, p.w_qkv, ep, rows, p.value_dtype,
                                      status, st, p.weights_settled)
                      : launch_qkv_rope_gemm(b.h, p.w_qkv, ep, rows, p.value_dtype, status, st, 1);
    if (rc != 0) return rc;
    if (few_tiles) {
      rc = launch_few_attn(b.q, b.k, b.v, ring_k, ring_v, b.core, B, T, past, slots, p.window, p.scale, value_fp16, status, st, 1);
      if (rc == 0 && cached && !few_attn_updates_ring(T)) rc = launch_ring_append(b.k, b.v, ring_k, ring_v, B, T, past, slots, st, 1);
    } else if (!cached) {
      rc = launch_band_attn_prefill(b.q, b.k, b.v, b.core, B, T, p.window, p.scale, value_fp16, status, st, 1);
    } else if (few) {
      rc = launch_stream_attn(b.q, b.k, b.v, ring_k, ring_v, b.core, B, T, past, slots, p.window, p.scale, value_fp16, status, st, 1);
    } else {
      if (delta > 0) {
        rc = launch_ring_linearize(ring_k, ring_v, b.k, b.v, b.k_lin, b.v_lin, B, T, delta, past, slots, st, 1);
        if (rc != 0) return rc;
        rc = launch_band_attn_chunk(b.q, b.k_lin, b.v_lin, b.core, B, T, delta + T, p.window, p.scale, value_fp16, status, st, 1);
      } else {
        rc = launch_band_attn_prefill(b.q, b.k, b.v, b.core, B, T, p.window, p.scale, value_fp16, status, st, 1);
      }
      if (rc != 0) return rc;
      rc = launch_ring_append(b.k, b.v, ring_k, ring_v, B, T, past, slots, st, 1);
    }
  }
  if (rc != 0) return rc;
  if (one_tail) {
    const LayerTail t = {b.core, p.w_o, p.w_fc1, p.w_fc2, x, y, vec(p.attn_scale), vec(p.mlp_scale), vec(p.ln2_weight), vec(p.ln2_bias),
                         p.ln2_eps, p.stream_dtype, value_fp16, tc, front ? 8 * B : 0};
    return launch_layer_tail(t, rows, status, st, 1);
  }
  rc = launch_linear_gemm(b.core, p.w_o, b.x1, vec(p.attn_scale), x, rows, 512, 512, value_fp16, p.stream_dtype, 0, status, st, 1);
  if (rc != 0) return rc;
  if (norm2_inside) {
    rc = launch_ln_linear_gelu(b.x1, p.stream_dtype, vec(p.ln2_weight), vec(p.ln2_bias), p.ln2_eps, p.w_fc1, b.g, rows, p.ffn, tc, status,
                               st, 1);
  } else {
    rc = launch_layernorm512(b.x1, p.stream_dtype, vec(p.ln2_weight), vec(p.ln2_bias), p.ln2_eps, b.h, tc, rows, st, 1);
    if (rc != 0) return rc;
    rc = launch_linear_gemm(b.h, p.w_fc1, b.g, ParamVec(nullptr), nullptr, rows, p.ffn, 512, tc, tc, 1, status, st, 1);
  }
  if (rc != 0) return rc;
  return launch_linear_gemm(b.g, p.w_fc2, y, vec(p.mlp_scale), b.x1, rows, 512, p.ffn, tc, p.stream_dtype, 0, status, st, 1);
}

}  // namespace fm

extern "C" int fm_layer_forward(const fm_layer_params* params, const void* x, void* y, void* workspace,
                                long long workspace_bytes, const float* cos, const float* sin, long long cos_bstride, int B,
                                int T, void* ring_k, void* ring_v, int past, int ring_slots, int* status, void* stream) {
  if (params == nullptr || params->stream_dtype < 0 || params->stream_dtype > 2 || params->value_dtype < 0 ||
      params->value_dtype > 3 || params->vec_dtype < 0 || params->vec_dtype > 2 ||
      (params->stream_dtype == 2 && params->vec_dtype != 2))
    return -1;
  return fm::layer_forward(*params, x, y, workspace, workspace_bytes, cos, sin, cos_bstride, B, T, ring_k, ring_v, past,
                           ring_slots, status, static_cast<cudaStream_t>(stream));
}
