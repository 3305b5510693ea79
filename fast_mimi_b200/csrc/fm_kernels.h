// Internal launcher declarations shared by the .cu files of the library.
//
// `dependent`: the launch may start before the kernel in front of it has finished (programmatic dependent launch).  Only
// for kernels launched behind one another by one entry point: the first kernel of such a chain reads nothing before its
// wait, so what the later ones read early (weights, rows already in a ring) was complete before the chain began.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fm_common.cuh"

namespace fm {

// Whether one of a call's tensors has no memory.  A kernel would fault on it; a tensor that only stands for one (a fake one of
// torch's) says that it lies on the device and has address 0.
template <typename... P>
inline bool absent(const P*... p) { return (... || (p == nullptr)); }

// Where the projection epilogue puts its results.  Linear outputs are [M, 512] 16-bit tensors
// (null = skip).  The KV ring is [clips, 8 heads, ring_slots, 64]; the frame at absolute position
// p of a clip lands in slot p % ring_slots.
struct QkvEpilogueArgs {
  uint16_t* q;
  uint16_t* k;
  uint16_t* v;
  uint16_t* ring_k;
  uint16_t* ring_v;
  const float* cos;        // [1 or clips, T, 64] FP32, as the reference's position_embeddings
  const float* sin;
  long long cos_bstride;   // 0 (one table for all clips) or T*64
  const int* clip_pos;     // optional device array: absolute position of frame 0 of each clip
  int pos_base;            // added to every position
  int T;                   // frames per clip in this call
  int ring_slots;
  // Output projection mode (launch_out_proj_gemm): the weight has two 256-wide output tiles instead of
  // six, results go out through `v` without RoPE as  resid + out_scale[c] * acc  (both optional).
  int n_tiles;             // 256-wide output tiles of the weight: 6 (q|k|v) or 2 (one 512-wide output)
  int seg_base;            // segment of output tile 0: 0 (q, k, v in turn) or 2 (plain output)
  const float* out_scale;  // [512] per-channel factor (the reference's layer scale) or null
  const uint16_t* resid;   // [M, 512] residual in the output's 16-bit format or null
};

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time libcuda).
int encode_tiled(CUtensorMap* map, CUtensorMapDataType dtype, uint32_t rank, void* base, const cuuint64_t* dims,
                 const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* elem_strides,
                 CUtensorMapSwizzle swizzle);
// [rows, cols] row-major 16-bit matrix, boxes of box_rows x box_cols, 128-byte swizzle.
int encode_rows_16bit(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols);
// The projection kernels read the rotary tables four values at a time.
inline bool rope_tables_aligned(const float* cos, const float* sin, long long bstride) {
  return ((reinterpret_cast<uintptr_t>(cos) | reinterpret_cast<uintptr_t>(sin) | static_cast<uintptr_t>(bstride) * sizeof(float)) & 15u) == 0;
}
// Multiprocessors of the current device.
int sm_count();
// Opt a kernel into `bytes` of dynamic shared memory once per (kernel, device).
int ensure_dynamic_smem(const void* kernel, int bytes);

int launch_linear_fp32(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t st);
int launch_rope_fp32(float* t, const float* cosv, const float* sinv, int B, int T, int H, int D,
                     long long cos_bstride, cudaStream_t st);
int launch_band_attn_fp32(const float* q, const float* k, const float* v, float* out, int B, int H, int D,
                          int Tq, int Tk, int q_off, int k_off, int window, float scale,
                          const long long* strides, cudaStream_t st);
int launch_qkv_rope_gemm(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags,
                         int* status, cudaStream_t st, int dependent = 0);
// y[M,512] = resid + out_scale * (a[M,512] * w[512,512]^T): the attention output projection with the layer
// scale and the residual add of the reference's transformer layer folded into the epilogue.
int launch_out_proj_gemm(const void* a, const void* w, void* y, const float* out_scale, const void* resid, int M,
                         int dtype_flags, int* status, cudaStream_t st);
// y[M,N] = resid + scale * act(a[M,K] * w[N,K]^T); in_dtype 0 BF16 / 1 FP16; out_dtype 0 BF16 / 1 FP16 / 2 FP32
// (type of y and resid); gelu 1 = exact GELU.  N a multiple of 256, K a multiple of 64.
int launch_linear_gemm(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N,
                       int K, int in_dtype, int out_dtype, int gelu, int* status, cudaStream_t st, int dependent = 0);
// Split-precision product y = (a_hi + a_lo)(w_hi + w_lo)^T in FP32 grade (all four FP16; lo lo left out).  `a` is [a_rows,
// a_cols]; row r of the product has K = a_cols * n values and lies in rows r .. r + n - 1 of `a` (n = 1: a plain matrix; n = 2:
// a convolution of twice its stride over padded frames).  Of every clip_rows rows the first clip_valid are results, stored
// back to back: y [rows * clip_valid / clip_rows, N]; or, with by_channel, clip by clip with the channels outside: y
// [rows / clip_rows, N, clip_valid].  n_mats > 1: y is so many matrices [.., N / n_mats], one behind the other (several weights'
// products with the same rows).  parts = 2: the two halves of K are products of their own (two matrices side by side), whose
// sums are added once in FP32.  Together in one accumulator they lose bits that two products do not: the tensor core cuts
// every addend to the accumulator's exponent (K = 512 as one sum 7.0e-7 of the result against 64 bits, as two of 256 4.5e-7).
struct SplitRows {
  int a_chunks;           // a_cols / 64
  int clip_rows, clip_valid;
  int by_channel;
  int parts;              // K ranges that have an accumulator each, added in FP32: 1 or 2
  int cols;               // N / n_mats
  long long mat_step;     // values of one of the matrices
  // where column `col` (of a tile that lies in one matrix) of result row `row` goes
  __host__ __device__ __forceinline__ long long at(int row, int col) const {
    const int mat = col / cols;
    return mat * mat_step + static_cast<long long>(row) * cols + (col - mat * cols);
  }
  __host__ __device__ __forceinline__ int out_row(int row, int M) const {
    if (row >= M) return -1;
    if (clip_rows == clip_valid) return row;
    const int clip = row / clip_rows, t = row - clip * clip_rows;
    return t < clip_valid ? clip * clip_valid + t : -1;
  }
  // channel 0 of a row in the by_channel layout; channels are clip_valid values apart
  __host__ __device__ __forceinline__ long long out_at(int row, int M, int N) const {
    const int clip = row / clip_rows, t = row - clip * clip_rows;
    return row < M && t < clip_valid ? static_cast<long long>(clip) * N * clip_valid + t : -1;
  }
};
// The K chunks of a split-precision product in the order of its sums: part by part, in a part lo W_hi, hi W_lo, hi W_hi (the
// small terms first).
struct SplitWalk {
  int part_chunks;        // K chunks of a part in one term
  int part, term, k;      // k: chunk of the operands
  __device__ __forceinline__ SplitWalk(int chunks, int index) : part_chunks(chunks), part(index / (3 * chunks)) {
    const int left = index - 3 * chunks * part;
    term = left / chunks;
    k = part * chunks + left - term * chunks;
  }
  __device__ __forceinline__ bool a_low() const { return term == 0; }
  __device__ __forceinline__ bool w_low() const { return term == 1; }
  __device__ __forceinline__ void next() {
    if (++k < (part + 1) * part_chunks) return;
    if (++term == 3) {
      term = 0;
      ++part;
    }
    k = part * part_chunks;
  }
};
// Tensor maps of the lo parts: a kernel argument of split-precision products alone (256 bytes more cost every launch of the
// others a quarter of a microsecond).
template <bool kSplit> struct SplitMaps {};
template <> struct SplitMaps<true> { CUtensorMap a, w; };
struct SplitLow {
  const void *a, *w;
  long long a_rows;
};
int launch_linear_split(const void* a_hi, const void* a_lo, long long a_rows, int a_cols, const void* w_hi, const void* w_lo, float* y,
                        long long rows, int clip_rows, int clip_valid, int by_channel, int n_mats, int parts, int N, int K, int* status,
                        cudaStream_t st, int dependent = 0);
int launch_linear_split_small(const void* a_hi, const void* w_hi, const SplitLow& low, const SplitRows& map, float* y, int M, int N,
                              int K, int* status, cudaStream_t st, int dependent);
// The same from an operand as it lies, split on the way (fm_split_gemm.cu), for many rows: FP32 rows [rows, K], or frames [B, T, C] of
// a causal convolution.  K a multiple of 128, at least 256.
// Whether there are rows enough for them to be the faster form.
bool split_gemm_takes(long long rows, int N, int K);
int launch_split_rows(const float* x, const void* w_hi, const void* w_lo, float* y, long long rows, int n_mats, int N, int K, int* status,
                      cudaStream_t st);
int launch_split_conv(const float* x, const void* w_hi, const void* w_lo, float* y, int B, int T, int C, int kernel, int stride, int N, int* status,
                      cudaStream_t st);
// Padded frames of a causal convolution (kernel a multiple of stride), split into FP16 hi + lo parts: clip b has
// stride * (ceil(T / stride) + kernel / stride - 1) frames of C values (fm_downsample.cu).
int launch_conv_frames_split(const float* x, void* hi, void* lo, int B, int T, int C, int kernel, int stride, cudaStream_t st);
// The same two products for few rows (fm_linear_small.cu): 128 x 64 tiles, K split over a cluster.
bool few_row_tiles(int M, int N);
// LayerNorm folded into the product behind it (fm_ln_linear.cu) while one wave of blocks holds the rows: the chain-opening QKV projection and
// gelu(LayerNorm(x) W^T).
bool few_rows_with_norm(int M, int N);
int launch_ln_qkv(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, const void* w_qkv,
                  const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status, cudaStream_t st, int dependent);
int launch_ln_linear_gelu(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, const void* w, void* y,
                          int M, int N, int tc_fp16, int* status, cudaStream_t st, int dependent);
int launch_linear_small(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N, int K,
                        int in_dtype, int out_dtype, int gelu, int* status, cudaStream_t st, int dependent);
// The same for as few rows as one wave of blocks with their weights in tensor memory holds (fm_linear_ws.cu): K a power of two times 512.
bool linear_ws_takes(int M, int N, int K, int dependent, bool resid16 = false);      // resid16: onto a residual of 16 bits
int launch_linear_ws(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N, int K, int in_dtype, int out_dtype, int gelu,
                     int* status, cudaStream_t st, int dependent);
int launch_qkv_ws(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status, cudaStream_t st,
                  int dependent);
int launch_qkv_small(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status,
                     cudaStream_t st, int dependent);
// Output projection, LayerNorm and MLP of a layer in one kernel (fm_layer_tail.cu), for as many rows as layer_tail_takes says:
// y = x1 + mlp_scale * (gelu(LayerNorm(x1) w_fc1^T) w_fc2^T),  x1 = x + attn_scale * (core w_o^T).  A scale without data: one.
struct LayerTail {
  const void *core, *w_o, *w_fc1, *w_fc2;    // [M, 512] and [512, 512] of the value type; [2048, 512] and [512, 2048] of the MLP's
  const void* x;                             // [M, 512] of stream_type (0 BF16, 1 FP16, 2 FP32), like y
  void* y;
  ParamVec attn_scale, mlp_scale, ln_weight, ln_bias;
  float eps;
  int stream_type, value_fp16, tc_fp16;
  int beside;                                // blocks of the kernel in front that have an SM each to themselves
};
bool layer_tail_takes(int M, int ffn);
int launch_layer_tail(const LayerTail& t, int M, int* status, cudaStream_t st, int dependent);
// LayerNorm over 512 channels; x_dtype 0 BF16 / 1 FP16 / 2 FP32, y_dtype 0 BF16 / 1 FP16.
int launch_layernorm512(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, void* y,
                        int y_dtype, long long rows, cudaStream_t st, int dependent = 0);
// Residual vector quantisation (fm_rvq.cu): candidate selection + exact FP32 decision for one layer, FP16 copy of
// the residual, ordered FP32 decode.
int launch_rvq_select(const void* scores, int scores_fp16, const float* e_sq, const float* codebook, float* resid, void* resid16,
                      long long* codes, int* n_candidates, long long rows, int n_codes, float e_max, float tau_rel,
                      int* status, cudaStream_t st);
// Rows of a strided causal convolution with replicate padding, gathered from frame-major FP32 activations and split
// into FP16 hi + lo parts: [B * ceil(T / stride), kernel * C] (fm_downsample.cu).
int launch_conv_rows_split(const float* x, void* hi, void* lo, int B, int T, int C, int kernel, int stride,
                           cudaStream_t st);
int launch_wait_timeout_selftest(int* status, int limit_us, int* observed, cudaStream_t st);
// y[B, 2T, C] from x[B, T, C] by the depthwise transposed convolution of kernel 4, stride 2 (w [C, 4]), FP32.
int launch_upsample2_depthwise(const float* x, const float* w, float* y, int B, int T, int C, cudaStream_t st);
int launch_split_half(const float* x, void* hi, void* lo, long long n, cudaStream_t st);
// Record-based variant (no scores in memory): candidate records from launch_linear_gemm(out_dtype 3), per-frame
// margins in `tau` (written for the next layer by the decision kernel, for the first layer by launch_rvq_prepare).
int launch_rvq_select_rec(const void* records, const float* codebook, float* resid, void* resid16, long long* codes,
                          int* n_candidates, float* tau, long long rows, int n_codes, float e_max_next, float tau_rel,
                          int* status, cudaStream_t st, int dependent = 0, int last = 0);
int launch_rvq_encode(float* resid, void* resid16, float* tau, void* records, const void* books16, const float* books, const float* e_sq,
                      const float* e_max, long long* codes, int* n_candidates, long long rows, int n_codes, int layers, float tau_rel,
                      int* status, cudaStream_t st);
// One or two stacks over vectors of their own, the same number of them and of entries per codebook.
struct RvqStack {
  float* residual;        // [rows, 256], overwritten
  const void* books16;    // [layers, n_codes, 256] FP16, FP32
  const float *books, *e_sq, *e_max;      // e_max [layers] in host memory
  long long* codes;       // [layers, rows]
  int layers;
};
int launch_rvq_encode_stacks(const RvqStack* stacks, int n_stacks, void* resid16, float* tau, void* records, long long rows, int n_codes,
                             float tau_rel, int* status, cudaStream_t st);
// The whole search in one kernel for many vectors (fm_rvq_tiles.cu); the workspaces are left alone.
bool rvq_tiles_take(const RvqStack* stacks, int n_stacks, long long rows, int n_codes);
int launch_rvq_tiles(const RvqStack* stacks, int n_stacks, long long rows, int n_codes, float tau_rel, int* status, cudaStream_t st);
// The whole search in one kernel for few vectors (fm_rvq_stack.cu); nothing but codes is written.
bool rvq_stack_takes(const RvqStack* stacks, int n_stacks, long long rows, int n_codes);
// With `from` the vectors are projected on the way: x [rows, 512], w_hi and w_lo [256 n_stacks, 512]; `residual` is not looked at.
struct RvqFrames {
  const float* x;
  const void *w_hi, *w_lo;
};
int launch_rvq_stack(const RvqStack* stacks, int n_stacks, long long rows, float tau_rel, int* status, cudaStream_t st,
                     const RvqFrames* from = nullptr);
int launch_rvq_prepare(const float* x, void* resid16, float* tau, long long rows, float e_max, float tau_rel,
                       cudaStream_t st);
int launch_rvq_to_half(const float* x, void* y, long long rows, cudaStream_t st);
// Ordered sums of one or two stacks (the first n0 of the n_layers rows of codes [B, n_layers, T]; the rest) as FP16 hi + lo
// parts [B * T, 256 or 512].
int launch_rvq_decode_split(const long long* codes, const float* books0, const float* books1, void* hi, void* lo, int B, int T,
                            int n_layers, int n0, int n_codes0, int n_codes1, int* bad_code, cudaStream_t st);
// The upsampling from [B, C, T] (fm_downsample.cu).
int launch_upsample2_channels(const float* x, const float* w, float* y, int B, int T, int C, cudaStream_t st);
int launch_rvq_decode(const long long* codes, const float* codebooks, float* out, long long rows, int n_layers,
                      int n_codes, int* bad_code, cudaStream_t st);
int launch_band_attn_prefill(const void* q, const void* k, const void* v, void* out, int B, int T, int window,
                             float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent = 0);
// Queries [B, Tq, 512] against keys / values [B, Tk, 512], Tk >= Tq: the last Tq key rows are the queries' own
// frames, the Tk - Tq rows before them are older (cached) frames.
int launch_band_attn_chunk(const void* q, const void* k, const void* v, void* out, int B, int Tq, int Tk, int window,
                           float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent = 0);
// KV ring <-> frame-major tensors for multi-frame cached calls (fm_ring.cu).
int launch_ring_linearize(const void* ring_k, const void* ring_v, const void* k_new, const void* v_new, void* k_lin,
                          void* v_lin, int S, int T, int delta, int past, int slots, cudaStream_t st, int dependent = 0);
int launch_ring_append(const void* k_new, const void* v_new, void* ring_k, void* ring_v, int S, int T, int past,
                       int slots, cudaStream_t st, int dependent = 0);
// T <= 8 new frames per stream over its ring (at most 256 slots), ring update included (fm_stream_attn.cu).
int launch_stream_attn(const void* q, const void* k, const void* v, void* ring_k, void* ring_v, void* out, int S, int T,
                       int past, int slots, int window, float scale, int value_is_fp16, int* status, cudaStream_t st,
                       int dependent = 0);
// LayerNorm, projection and that attention in one kernel (fm_stream_front.cu), which opens a layer's chain, for as many streams as
// stream_front_takes says.
struct StreamFront {
  const void* x;                  // [S, T, 512] of stream_type
  ParamVec ln_weight, ln_bias;
  float eps;
  const void* w_qkv;
  const float *cos, *sin;
  long long cos_bstride;
  void *ring_k, *ring_v, *core;
  int stream_type, value_fp16, tc_fp16;
};
bool stream_front_takes(int S, int T, int slots);
int launch_stream_front(const StreamFront& f, int S, int T, int past, int slots, int window, float scale, int* status, cudaStream_t st, int dependent);
// Attention for few query tiles (fm_few_attn.cu): at most two 64-query blocks per SM.  ring_k null: clips; else T new frames
// per stream on top of the ring, which the kernel also updates with up to 64 of them.
bool few_attn_tiles(int S, int T);
bool few_attn_updates_ring(int T);
int launch_few_attn(const void* q, const void* k, const void* v, void* ring_k, void* ring_v, void* out, int S, int T, int past,
                    int slots, int window, float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent = 0);
// Projection + RoPE + banded attention in one kernel for 128 < T <= 256 (fm_fused_clip.cu): q, k, v stay on chip.
int launch_attn_fused_clip(const void* x, const void* w_qkv, const float* cos, const float* sin, long long cos_bstride,
                           void* out, int B, int T, int window, float scale, int dtype_flags, int* status,
                           cudaStream_t st, int dependent = 0);
// Whether whole clips take the one-kernel form (fm_fused_clip.cu) rather than projection + attention.
bool use_fused_clip(int B, int T);
int launch_band_attn_clip(const void* q, const void* k, const void* v, void* out, int B, int T, int window,
                          float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent = 0);
// out_fp32: out is FP32 (else the value type)
int launch_band_attn_long(const void* q, const void* k, const void* v, void* out, int B, int T, int window,
                          float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent = 0, int out_fp32 = 0);
bool band_attn_long_takes(int T, int window);
// The same on FP32 q, k, v [B, 8, T, 64] of the given strides (three of each, in values: clip, head, frame), FP32 result.
bool band_attn_long_takes_f32(const long long* strides, int B, int T);
int launch_band_attn_long_f32(const void* const* qkv, const long long* strides, float* out, int B, int T, int window, float scale,
                              int value_is_fp16, int* status, cudaStream_t st);
// Banded attention on [B, 8, T, 64] tensors of any float type and strides (fm_window.cu).
int launch_window_attention(const void* const* qkv, int in_type, const long long* strides, void* const* ws, void* out16, float* out32,
                            int B, int T, int window, float scale, int value_is_fp16, int* status, cudaStream_t st);
int launch_ring_decode_attn(const void* q, const void* ring_k, const void* ring_v, float* out,
                            const int* stream_pos, int pos_base, int S, int ring_slots, float scale,
                            int value_is_fp16, int* status, cudaStream_t st);

}  // namespace fm
