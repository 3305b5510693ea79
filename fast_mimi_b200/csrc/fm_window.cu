// Banded attention on q, k, v as a model holds them (sm_100a): any of FP32, BF16 and FP16, [B, 8, T, 64] with any strides and a
// contiguous last dimension (reference: _native_window_attention, src/fast_mimi/model.py:1589-1624).
//
// The attention kernels read frame-major 16-bit tensors.  The kernel for long clips rounds FP32 tensors itself on the way in where its
// blocks have some steps each, whatever the strides, as far as a tensor map can have them (fm_prefill_long.cu: 16 clips of 2500 frames 105 us,
// 135 with a converting pass in front).  For the others bringing FP32 inputs there is HBM-bound: 12 bytes read and six
// written per value triple, one launch for the three.  The way back is free where the kernel for long clips stores FP32 (a
// converting pass over the result took 51 us).
#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"

namespace fm {

namespace window {
struct Job {
  const void* src;
  uint16_t* dst;
  long long sb, sh, st;      // strides in values
  int out_fp16;
};
struct Jobs {
  Job job[3];
};

__device__ __forceinline__ void load8(const void* src, long long at, int type, float (&v)[8]) {
  if (type == 2) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(src) + at);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(src) + at));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = type == 1 ? Pack16<__half>::unpack(w[e]) : Pack16<__nv_bfloat16>::unpack(w[e]);
      v[2 * e] = f.x;
      v[2 * e + 1] = f.y;
    }
  }
}
}  // namespace window

// blockIdx.y: the tensor; a thread converts two pieces of eight values.
__global__ void __launch_bounds__(256)
window_inputs_kernel(const __grid_constant__ window::Jobs jobs, int in_type, int T, long long pieces) {
  using namespace window;
  griddep_launch();
  const Job& j = jobs.job[blockIdx.y];
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < pieces; i += 2 * step) {
    float v[2][8];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const long long p = i + k * step;
      if (p < pieces) {
        const long long frame = p >> 6, b = frame / T;
        load8(j.src, b * j.sb + (frame - b * T) * j.st + ((p >> 3) & 7) * j.sh + (p & 7) * 8, in_type, v[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const long long p = i + k * step;
      if (p < pieces) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = j.out_fp16 ? Pack16<__half>::pack(v[k][2 * e], v[k][2 * e + 1]) : Pack16<__nv_bfloat16>::pack(v[k][2 * e], v[k][2 * e + 1]);
        reinterpret_cast<uint4*>(j.dst)[p] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// 16-bit result -> FP32, eight values per thread.
__global__ void __launch_bounds__(256)
window_output_kernel(const uint16_t* __restrict__ src, float* __restrict__ dst, int is_fp16, long long pieces) {
  griddep_wait();
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < pieces; i += step) {
    const uint4 u = __ldcg(reinterpret_cast<const uint4*>(src) + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float2 f[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = is_fp16 ? Pack16<__half>::unpack(w[e]) : Pack16<__nv_bfloat16>::unpack(w[e]);
    reinterpret_cast<float4*>(dst)[2 * i] = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
    reinterpret_cast<float4*>(dst)[2 * i + 1] = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
  }
}

int launch_window_attention(const void* const* qkv, int in_type, const long long* strides, void* const* ws, void* out16, float* out32,
                            int B, int T, int window_size, float scale, int value_is_fp16, int* status, cudaStream_t st) {
  using namespace window;
  if (B <= 0 || T <= 0) return (B == 0 || T == 0) ? 0 : -1;
  if (in_type < 0 || in_type > 2 || B > 65535) return -1;
  const uint64_t vec = in_type == 2 ? 4 : 8;          // values per 16 bytes
  Jobs jobs = {};
  const void* in16[3];
  unsigned n = 0;
  for (int i = 0; i < 3; ++i) {
    const long long* s = strides + 3 * i;
    if (qkv[i] == nullptr || (reinterpret_cast<uintptr_t>(qkv[i]) & 15u) != 0) return -3;
    if (ws[i] == nullptr) {                            // already frame-major and of the attention's type
      if (in_type != (i == 2 ? value_is_fp16 : 0) || s[1] != 64 || s[2] != 512 || (B > 1 && s[0] != 512ll * T)) return -1;
      in16[i] = qkv[i];
      continue;
    }
    if ((static_cast<uint64_t>(s[0]) | static_cast<uint64_t>(s[1]) | static_cast<uint64_t>(s[2])) % vec != 0 ||
        (reinterpret_cast<uintptr_t>(ws[i]) & 15u) != 0)
      return -3;
    jobs.job[n++] = {qkv[i], static_cast<uint16_t*>(ws[i]), s[0], s[1], s[2], i == 2 ? value_is_fp16 : 0};
    in16[i] = ws[i];
  }
  const bool direct = out32 != nullptr && band_attn_long_takes(T, window_size);
  const bool converts = direct && in_type == 2 && band_attn_long_takes_f32(strides, B, T);     // the attention kernel itself
  if ((reinterpret_cast<uintptr_t>(out16) | reinterpret_cast<uintptr_t>(out32)) & 15u) return -3;
  if (!direct && out16 == nullptr) return -1;
  if (converts) return launch_band_attn_long_f32(qkv, strides, out32, B, T, window_size, scale, value_is_fp16, status, st);
  const long long pieces = static_cast<long long>(B) * T * 64;
  const auto blocks = [&](long long threads) {
    const long long want = (threads + 255) / 256, cap = static_cast<long long>(sm_count()) * 8;
    return static_cast<unsigned>(want < cap ? want : cap);
  };
  int rc = 0;
  if (n > 0) rc = launch_kernel(window_inputs_kernel, dim3(blocks((pieces + 1) / 2), n), 256, 0, st, 1, 0, jobs, in_type, T, pieces);
  if (rc != 0) return rc;
  if (direct)
    return launch_band_attn_long(in16[0], in16[1], in16[2], out32, B, T, window_size, scale, value_is_fp16, status, st, n > 0, 1);
  rc = launch_band_attn_prefill(in16[0], in16[1], in16[2], out16, B, T, window_size, scale, value_is_fp16, status, st, n > 0);
  if (rc != 0 || out32 == nullptr) return rc;
  return launch_kernel(window_output_kernel, dim3(blocks(pieces)), 256, 0, st, 1, 1, static_cast<const uint16_t*>(out16), out32,
                       value_is_fp16, pieces);
}

}  // namespace fm
