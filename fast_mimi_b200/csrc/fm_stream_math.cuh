// What the kernels of live streams share (fm_stream_attn.cu, fm_stream_front.cu).
#pragma once

#include "fm_common.cuh"

namespace fm {

// Probabilities as operands of type T without losing bits of FP32: as a sum of kParts values.  BF16 has eight significant bits
// and the range of FP32: three parts are all 24.  FP16 has eleven, and a sign on the second part makes two of them 24 to within
// the last bit, but nothing below 2^-24: probabilities carry a factor of 2^kShift, the sum they are divided by likewise.  (As two
// parts each and unscaled, an FP16 result carried by probabilities of 2^-20 was off by up to 4e-3, one of BF16 by 2^-17 of its terms.)
template <typename T> struct Parts { static constexpr int kParts = 3; static constexpr float kShift = 0.f; };
template <> struct Parts<__half> { static constexpr int kParts = 2; static constexpr float kShift = 15.f; };

template <typename T>
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&part)[Parts<T>::kParts]) {
#pragma unroll
  for (int i = 0; i < Parts<T>::kParts; ++i) {
    part[i] = Pack16<T>::pack(x, y);
    const float2 b = Pack16<T>::unpack(part[i]);
    x -= b.x;
    y -= b.y;
  }
}

}  // namespace fm
