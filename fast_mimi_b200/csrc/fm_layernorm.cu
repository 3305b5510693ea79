// LayerNorm over the 512-wide hidden dimension, written for the activations that feed the tensor-core
// projections: input in FP32, FP16 or BF16, output rounded once to FP16 or BF16.
//
// Replaces nn.LayerNorm(hidden_size, eps) in front of the attention and MLP branches of the reference's
// transformer layer (src/fast_mimi/model.py:2021-2024, applied at :2052 and :2060): biased variance,
// (x - mean) * rsqrt(var + eps) * weight + bias, all in FP32.
//
// One warp per frame: each lane holds 16 values (four 4-element pieces, 32 lanes apart, so every load and
// store instruction of the warp touches one contiguous run), two shuffle reductions, no shared memory.
// HBM-bound: reads the frame once, writes it once.
#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"

namespace fm {

namespace ln {
constexpr int kHidden = 512;
constexpr int kWarpsPerBlock = 8;

}  // namespace ln

// Four weights (or biases) as they lie and as FP32.  16-bit ones stay packed until they are used: 16 registers less.
template <int kVec> struct Vec4;
template <> struct Vec4<2> {
  float4 v;
  __device__ __forceinline__ void load(const ParamVec& p, int i) { v = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p.data) + i)); }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <int kVec> struct Vec4 {
  using T16 = typename std::conditional<kVec == 1, __half, __nv_bfloat16>::type;
  uint2 u;
  __device__ __forceinline__ void load(const ParamVec& p, int i) { u = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.data) + i)); }
  __device__ __forceinline__ float4 get() const {
    const float2 a = Pack16<T16>::unpack(u.x), b = Pack16<T16>::unpack(u.y);
    return make_float4(a.x, a.y, b.x, b.y);
  }
};

// HBM-bound, so what counts is bytes in flight: four blocks of 64 registers per SM, hence the bound.  (Asking for the next
// frame at the end of an iteration, with weights of any type behind a test, took 80 registers and three blocks: 128000 frames of
// BF16 52.9 us against 45.2, 16000 of FP32 6.5 against 5.7; 64 clips of 10 s through four BF16 layers 549 against 532.)
// kIn, kVec (type of weight and bias): 0 = BF16, 1 = FP16, 2 = FP32;  kOut: 0 = BF16, 1 = FP16
template <int kIn, int kOut, int kVec>
__global__ void __launch_bounds__(ln::kWarpsPerBlock * 32, 4)
layernorm512_kernel(const void* __restrict__ x, const ParamVec weight, const ParamVec bias,
                    float eps, void* __restrict__ y, long long rows) {
  using namespace ln;
  using TOut = typename std::conditional<kOut == 1, __half, __nv_bfloat16>::type;
  // This kernel opens a layer's chain of dependent launches: it lets the next kernel start only after its own wait, so
  // whatever that one reads ahead of ITS wait (weights) was complete before the chain began.
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31;
  const long long warp0 = static_cast<long long>(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5);
  const long long stride = static_cast<long long>(gridDim.x) * kWarpsPerBlock;
  // this lane's channels: 4*lane + 128*j + (0..3); weight and bias stay in registers across frames
  Vec4<kVec> w[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[j].load(weight, 128 * j + 4 * lane);
    b[j].load(bias, 128 * j + 4 * lane);
  }
  for (long long row = warp0; row < rows; row += stride) {
    float v[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) load4<kIn>(x, row * kHidden + 128 * j + 4 * lane, v[j]);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) sum += (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum * (1.0f / kHidden);
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[j][e] -= mean;
        sq += v[j][e] * v[j][e];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq * (1.0f / kHidden) + eps);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 wf = w[j].get(), bf = b[j].get();
      const float o[4] = {v[j][0] * rstd * wf.x + bf.x, v[j][1] * rstd * wf.y + bf.y, v[j][2] * rstd * wf.z + bf.z,
                          v[j][3] * rstd * wf.w + bf.w};
      const uint2 packed = make_uint2(Pack16<TOut>::pack(o[0], o[1]), Pack16<TOut>::pack(o[2], o[3]));
      *reinterpret_cast<uint2*>(static_cast<uint16_t*>(y) + row * kHidden + 128 * j + 4 * lane) = packed;
    }
  }
}

int launch_layernorm512(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, void* y,
                        int y_dtype, long long rows, cudaStream_t st, int dependent) {
  using namespace ln;
  if (rows < 0 || x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 1) return -1;
  if (weight.type < 0 || weight.type > 2 || bias.type != weight.type || (x_dtype == 2 && weight.type != 2)) return -1;
  if (rows == 0) return 0;
  if (x == nullptr || y == nullptr || weight.data == nullptr || bias.data == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(weight.data) |
       reinterpret_cast<uintptr_t>(bias.data)) & 15u)
    return -3;
  const long long want = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const long long cap = static_cast<long long>(sm_count()) * 4;    // resident blocks: 256 threads of 64 registers
  const int grid = static_cast<int>(want < cap ? want : cap);
  using Kern = void (*)(const void*, ParamVec, ParamVec, float, void*, long long);
  static const Kern table[7][2] = {
      {layernorm512_kernel<0, 0, 0>, layernorm512_kernel<0, 1, 0>}, {layernorm512_kernel<0, 0, 1>, layernorm512_kernel<0, 1, 1>},
      {layernorm512_kernel<0, 0, 2>, layernorm512_kernel<0, 1, 2>}, {layernorm512_kernel<1, 0, 0>, layernorm512_kernel<1, 1, 0>},
      {layernorm512_kernel<1, 0, 1>, layernorm512_kernel<1, 1, 1>}, {layernorm512_kernel<1, 0, 2>, layernorm512_kernel<1, 1, 2>},
      {layernorm512_kernel<2, 0, 2>, layernorm512_kernel<2, 1, 2>}};
  return launch_kernel(table[x_dtype == 2 ? 6 : 3 * x_dtype + weight.type][y_dtype], dim3(grid), kWarpsPerBlock * 32, 0, st, 1, dependent, x, weight, bias, eps, y,
                       rows);
}

}  // namespace fm
