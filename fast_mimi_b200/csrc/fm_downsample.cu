// The two stride-2 convolutions around the quantiser (sm_100a): `downsample` after the encoder transformer and
// `upsample` before the decoder transformer.
//
// Downsample.
// Reference: MimiModel.downsample = MimiConv1d(512 -> 512, kernel 4, stride 2, no bias, replicate padding, causal)
// (src/fast_mimi/model.py:2734-2744; forward of the class: left padding kernel - stride = 2 frames, right padding
// (-T) % 2 frames, both repeating the edge frame, then nn.Conv1d).  On frame-major activations [B, T, 512] output
// frame t is a 2048-long inner product: the four consecutive frames 2t-2 .. 2t+1 (clamped to the clip) against
// the kernel laid out as W2[c_out, j * 512 + c_in] = W[c_out, c_in, j].  So the convolution is a linear with
// K = 2048 over rows that overlap in memory.  This file lays the frames out with their padding and splits them into FP16
// hi + lo parts; the products run on the tensor-core linear kernel (hi W_hi + hi W_lo + lo W_hi with FP32 accumulation:
// FP32-grade accuracy, which the code decisions that follow need).
#include "fm_common.cuh"
#include "fm_kernels.h"

namespace fm {

// Padded frames, for a kernel that is a multiple of the stride: clip b has stride * (T_out + kernel / stride - 1) frames, the
// first kernel - stride and the odd last one repeating the edge.  Seen as rows of `stride` frames, output frame t is
// rows t .. t + kernel / stride - 1 of its clip, which the product reads as they lie: every frame is written once, and not
// kernel / stride times as in the gathered rows below.  HBM-bound: four bytes read and four written per value
// (128000 frames of 512: 85 us, 6.2 TB/s).
// One thread per 8 values.
__global__ void __launch_bounds__(256)
conv_frames_split_kernel(const float* __restrict__ x, uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int B, int T, int T_pad,
                         int left, int C) {
  griddep_launch();                        // opens a chain; the product behind it waits for its end
  const int c8 = C / 8;
  const long long total = static_cast<long long>(B) * T_pad * c8;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
    const long long r = i / c8;
    const int piece = static_cast<int>(i - r * c8);
    const int b = static_cast<int>(r / T_pad);
    int f = static_cast<int>(r - static_cast<long long>(b) * T_pad) - left;
    f = f < 0 ? 0 : (f > T - 1 ? T - 1 : f);
    const float4* src = reinterpret_cast<const float4*>(x + (static_cast<long long>(b) * T + f) * C + piece * 8);
    const float4 a = __ldg(src), c = __ldg(src + 1);
    uint4 h, l;
    split_half8(a, c, h, l);
    reinterpret_cast<uint4*>(hi)[i] = h;
    reinterpret_cast<uint4*>(lo)[i] = l;
  }
}

int launch_conv_frames_split(const float* x, void* hi, void* lo, int B, int T, int C, int kernel, int stride, cudaStream_t st) {
  if (B <= 0 || T <= 0) return (B == 0 || T == 0) ? 0 : -1;
  if (C <= 0 || C % 8 != 0 || stride <= 0 || kernel < stride || kernel % stride != 0 || kernel > 16 || absent(x, hi, lo)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15u) return -3;
  const int T_pad = stride * ((T + stride - 1) / stride + kernel / stride - 1);
  const long long want = (static_cast<long long>(B) * T_pad * (C / 8) + 255) / 256, cap = static_cast<long long>(sm_count()) * 8;
  conv_frames_split_kernel<<<static_cast<int>(want < cap ? want : cap), 256, 0, st>>>(
      x, static_cast<uint16_t*>(hi), static_cast<uint16_t*>(lo), B, T, T_pad, kernel - stride, C);
  return static_cast<int>(cudaGetLastError());
}

// One thread per 8 values of a gathered row: rows [B * T_out, 4 * C], x [B, T, C] FP32 (C a multiple of 8).
__global__ void __launch_bounds__(256)
conv_rows_split_kernel(const float* __restrict__ x, uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int B, int T,
                       int T_out, int C, int kernel, int stride) {
  const int c8 = C / 8;
  const long long total = static_cast<long long>(B) * T_out * kernel * c8;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
    const int piece = static_cast<int>(i % c8);
    long long r = i / c8;
    const int j = static_cast<int>(r % kernel);
    r /= kernel;
    const int t = static_cast<int>(r % T_out);
    const long long b = r / T_out;
    int f = t * stride + j - (kernel - stride);          // frame of the padded sequence, replicate at both ends
    f = f < 0 ? 0 : (f > T - 1 ? T - 1 : f);
    const float4* src = reinterpret_cast<const float4*>(x + (b * T + f) * C + piece * 8);
    const float4 a = __ldg(src), c = __ldg(src + 1);
    uint4 h, l;
    split_half8(a, c, h, l);
    reinterpret_cast<uint4*>(hi)[i] = h;
    reinterpret_cast<uint4*>(lo)[i] = l;
  }
}

int launch_conv_rows_split(const float* x, void* hi, void* lo, int B, int T, int C, int kernel, int stride,
                           cudaStream_t st) {
  if (B <= 0 || T <= 0) return (B == 0 || T == 0) ? 0 : -1;
  if (C <= 0 || C % 8 != 0 || kernel < stride || stride <= 0 || kernel > 16 || absent(x, hi, lo)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15u) return -3;
  const int T_out = (T + stride - 1) / stride;
  const long long total = static_cast<long long>(B) * T_out * kernel * (C / 8);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long want = (total + 255) / 256, cap = static_cast<long long>(sms > 0 ? sms : 1) * 8;
  conv_rows_split_kernel<<<static_cast<int>(want < cap ? want : cap), 256, 0, st>>>(
      x, static_cast<uint16_t*>(hi), static_cast<uint16_t*>(lo), B, T, T_out, C, kernel, stride);
  return static_cast<int>(cudaGetLastError());
}

// Upsample.  Reference: MimiModel.upsample = MimiConvTranspose1d(512 -> 512, kernel 4, stride 2, groups = 512, no bias)
// (src/fast_mimi/model.py:2745-2753; forward of the class: nn.ConvTranspose1d, then the last kernel - stride = 2
// output frames are trimmed, causal with trim_right_ratio 1).  With one channel per group it is elementwise: on
// frame-major activations  y[b, n, c] = w[c, n % 2] x[b, n / 2, c] + w[c, n % 2 + 2] x[b, n / 2 - 1, c]  for
// n = 0 .. 2T-1 (the second term absent for n < 2).  FP32 in, FP32 out, HBM-bound: 4 bytes read (each x value serves
// four outputs through L1 / L2) and 8 written per input value.
__global__ void __launch_bounds__(256)
upsample2_depthwise_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int B, int T,
                           int C) {
  const int c4 = C / 4;
  const long long total = static_cast<long long>(B) * 2 * T * c4;
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
    const int cq = static_cast<int>(i % c4);
    long long r = i / c4;
    const int n = static_cast<int>(r % (2 * T));
    const long long b = r / (2 * T);
    const int t = n >> 1, j = n & 1;
    const float4 a = __ldg(reinterpret_cast<const float4*>(x + (b * T + t) * C) + cq);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t > 0) p = __ldg(reinterpret_cast<const float4*>(x + (b * T + t - 1) * C) + cq);
    const float* wc = w + static_cast<long long>(cq) * 16;        // four channels x four taps
    float4 o;
    o.x = wc[j] * a.x + wc[j + 2] * p.x;
    o.y = wc[4 + j] * a.y + wc[4 + j + 2] * p.y;
    o.z = wc[8 + j] * a.z + wc[8 + j + 2] * p.z;
    o.w = wc[12 + j] * a.w + wc[12 + j + 2] * p.w;
    reinterpret_cast<float4*>(y + (b * 2 * T + n) * C)[cq] = o;
  }
}

// The same from channel-major x [B, C, T], in which the quantiser's decode leaves it: a tile of 32 frames (and the one in
// front) x 32 channels turns round in shared memory, so that both sides move whole lines and no transposed copy is made.
__global__ void __launch_bounds__(256)
upsample2_channels_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int T, int C) {
  __shared__ float tile[32][33];                      // [channel][frame t0 - 1 ..]; rows of 33 words fall on different banks
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = static_cast<int>(blockIdx.x) * 32, c0 = static_cast<int>(blockIdx.y) * 32;
  const long long b = blockIdx.z;
  // All loads before the first of them is stored, and none under a test of its own (frames past the end repeat the last one and are
  // not read): a block is one round trip to memory (64 clips of 125 frames, 512 channels 22.5 -> 16.4 us,
  // 512 clips 119 -> 76).
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __ldg(x + (b * C + c0 + warp + 8 * i) * T + (t0 + lane < T ? t0 + lane : T - 1));
  float before = 0.f;                                 // the frame before the tile, of this lane's channel
  if (warp == 0 && t0 > 0) before = __ldg(x + (b * C + c0 + lane) * T + t0 - 1);
  const float4 k = __ldg(reinterpret_cast<const float4*>(w) + c0 + lane);      // this lane's channel
#pragma unroll
  for (int i = 0; i < 4; ++i) tile[warp + 8 * i][lane + 1] = v[i];
  if (warp == 0) tile[lane][0] = before;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = warp + 8 * i;
    if (t0 + t >= T) break;
    const float p = tile[lane][t], a = tile[lane][t + 1];
    float* dst = y + (b * 2 * T + 2 * (t0 + t)) * C + c0 + lane;
    dst[0] = k.x * a + k.z * p;
    dst[C] = k.y * a + k.w * p;
  }
}

int launch_upsample2_channels(const float* x, const float* w, float* y, int B, int T, int C, cudaStream_t st) {
  if (B <= 0 || T <= 0) return (B == 0 || T == 0) ? 0 : -1;
  if (C <= 0 || C % 32 != 0 || B > 65535 || C / 32 > 65535 || absent(x, w, y)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) & 3u) | ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u)) return -3;
  const dim3 grid(static_cast<unsigned>((T + 31) / 32), static_cast<unsigned>(C / 32), static_cast<unsigned>(B));
  upsample2_channels_kernel<<<grid, 256, 0, st>>>(x, w, y, T, C);
  return static_cast<int>(cudaGetLastError());
}

int launch_upsample2_depthwise(const float* x, const float* w, float* y, int B, int T, int C, cudaStream_t st) {
  if (B <= 0 || T <= 0) return (B == 0 || T == 0) ? 0 : -1;
  if (C <= 0 || C % 4 != 0 || absent(x, w, y)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & 15u) return -3;
  const long long total = static_cast<long long>(B) * 2 * T * (C / 4);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long want = (total + 255) / 256, cap = static_cast<long long>(sms > 0 ? sms : 1) * 8;
  upsample2_depthwise_kernel<<<static_cast<int>(want < cap ? want : cap), 256, 0, st>>>(x, w, y, B, T, C);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fm
