// What the few-row product kernels share (fm_linear_small.cu, fm_ln_linear.cu): arguments, the layout of an FP32 tile of
// 64 columns in shared memory, and the epilogue of one piece of a finished row.
#pragma once

#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"

namespace fm {

namespace small {
// 16-byte piece `c` of FP32 row `r` of 64 (or 32) columns; the low three bits are permuted by `key`, the row's number in
// the tile, so that eight lanes with consecutive rows (writing) or consecutive pieces (reading) touch eight different
// bank groups.
template <int kCols = 64>
__device__ __forceinline__ uint32_t red_offset(uint32_t r, uint32_t c, uint32_t key) { return r * (kCols * 4u) + ((c ^ (key & 7u)) << 4); }
}  // namespace small

struct SmallArgs {
  ParamVec scale;         // [N] or null
  const void* resid;      // [M, N] in the output's type or null
  void* y;                // [M, N]
  int M, N, chunks;       // chunks: K / 64 / S, this block's share
  int split;              // S, blocks per cluster
  int gelu;
  QkvEpilogueArgs qkv;    // kOut 3
  SplitRows rows;         // kOut 4
  int part_chunks;        // kOut 4: K chunks of a part in one of the three products
};

// What the epilogue of eight values of row `row` of output tile `ntile` (64 columns, one attention head) reads besides the
// product: columns 4j .. 4j + 3 ([0]) and 32 + 4j .. ([1]), the two halves of RoPE pairs.  Asked for before the product
// is complete, so that its latency does not follow the reduction's.  With tiles of 32 columns (kHalves 1) a piece is four
// values.
// kOut: 0 = BF16, 1 = FP16, 2 = FP32 output and residual; 3 = q | k | v with RoPE; 4 = FP32 output of a split-precision product.
struct PieceOperands {
  float4 a[2];            // residual, or cos and sin
  uint4 s[2];             // per-channel scale, as it lies
};

template <int kOut, int kHalves = 2>
__device__ __forceinline__ void load_operands(const SmallArgs& args, int row, int ntile, int j, PieceOperands& p) {
  if constexpr (kOut == 3) {
    if (ntile < 16) {     // q and k
      const QkvEpilogueArgs& ep = args.qkv;
      const int clip = row / ep.T, t = row - clip * ep.T;
      const long long at = clip * ep.cos_bstride + static_cast<long long>(t) * 64 + 4 * j;
      p.a[0] = *reinterpret_cast<const float4*>(ep.cos + at);
      p.a[1] = *reinterpret_cast<const float4*>(ep.sin + at);
    }
  } else if constexpr (kOut != 4) {
    const int col = ntile * 32 * kHalves + 4 * j;
    const long long at = static_cast<long long>(row) * args.N + col;
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      if (args.scale.data != nullptr) p.s[h] = args.scale.raw4<kOut == 2>(col + 32 * h);
      p.a[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (args.resid != nullptr) {
        if constexpr (kOut == 2) {
          p.a[h] = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(args.resid) + at + 32 * h));
        } else {
          using T16 = typename std::conditional<kOut == 1, __half, __nv_bfloat16>::type;
          const uint2 r = __ldcg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(args.resid) + at + 32 * h));
          const float2 x = Pack16<T16>::unpack(r.x), y = Pack16<T16>::unpack(r.y);
          p.a[h] = make_float4(x.x, x.y, y.x, y.y);
        }
      }
    }
  }
}

// The epilogue itself: lo and hi are the product's columns 4j .. and 32 + 4j ..
template <int kOut, typename VT, int kHalves = 2>
__device__ __forceinline__ void finish_piece(const SmallArgs& args, float (&lo)[4], float (&hi)[4], const PieceOperands& p,
                                             int row, int ntile, int j, int* status) {
  if constexpr (kOut == 3) {
    const QkvEpilogueArgs& ep = args.qkv;
    const int seg = ntile >> 3, head = ntile & 7;
    uint2 plo, phi;
    if (seg < 2) {
      const float c[4] = {p.a[0].x, p.a[0].y, p.a[0].z, p.a[0].w}, sn[4] = {p.a[1].x, p.a[1].y, p.a[1].z, p.a[1].w};
      float o_lo[4], o_hi[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o_lo[e] = lo[e] * c[e] - hi[e] * sn[e];
        o_hi[e] = hi[e] * c[e] + lo[e] * sn[e];
      }
      plo = make_uint2(Pack16<__nv_bfloat16>::pack(o_lo[0], o_lo[1]), Pack16<__nv_bfloat16>::pack(o_lo[2], o_lo[3]));
      phi = make_uint2(Pack16<__nv_bfloat16>::pack(o_hi[0], o_hi[1]), Pack16<__nv_bfloat16>::pack(o_hi[2], o_hi[3]));
    } else {
      plo = make_uint2(Pack16<VT>::pack(lo[0], lo[1]), Pack16<VT>::pack(lo[2], lo[3]));
      phi = make_uint2(Pack16<VT>::pack(hi[0], hi[1]), Pack16<VT>::pack(hi[2], hi[3]));
    }
    uint16_t* lin = seg == 0 ? ep.q : (seg == 1 ? ep.k : ep.v);
    if (lin != nullptr) {
      uint16_t* dst = lin + static_cast<long long>(row) * 512 + head * 64 + 4 * j;
      *reinterpret_cast<uint2*>(dst) = plo;
      *reinterpret_cast<uint2*>(dst + 32) = phi;
    }
    uint16_t* ring = seg == 1 ? ep.ring_k : (seg == 2 ? ep.ring_v : nullptr);
    if (ring != nullptr) {
      const int clip = row / ep.T, t = row - clip * ep.T;
      const int pos = ep.pos_base + (ep.clip_pos != nullptr ? ep.clip_pos[clip] : 0) + t;
      if (pos < 0) {                     // would index another stream's ring: recorded, not written
        if (status != nullptr) atomicMax(status, static_cast<int>(kErrBounds));
      } else if (t >= ep.T - ep.ring_slots) {
        uint16_t* dst = ring + ((static_cast<long long>(clip) * 8 + head) * ep.ring_slots + pos % ep.ring_slots) * 64 + 4 * j;
        *reinterpret_cast<uint2*>(dst) = plo;
        *reinterpret_cast<uint2*>(dst + 32) = phi;
      }
    }
  } else if constexpr (kOut == 4) {
    if (args.rows.by_channel) {
      const long long at = args.rows.out_at(row, args.M, args.N), step = args.rows.clip_valid;
      if (at < 0) return;
      float* y = static_cast<float*>(args.y) + at + (ntile * 32 * kHalves + 4 * j) * step;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        y[e * step] = lo[e];
        if constexpr (kHalves == 2) y[(32 + e) * step] = hi[e];
      }
      return;
    }
    const int out = args.rows.out_row(row, args.M);
    if (out < 0) return;
    float* y = static_cast<float*>(args.y) + args.rows.at(out, ntile * 32 * kHalves + 4 * j);
    *reinterpret_cast<float4*>(y) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    if constexpr (kHalves == 2) *reinterpret_cast<float4*>(y + 32) = make_float4(hi[0], hi[1], hi[2], hi[3]);
  } else {
    const long long at = static_cast<long long>(row) * args.N + ntile * 32 * kHalves + 4 * j;
    float* part[2] = {lo, hi};
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      float* v = part[h];
      if (args.gelu) {
        gelu_erf2(v[0], v[1]);
        gelu_erf2(v[2], v[3]);
      }
      if (args.scale.data != nullptr) {
        const float4 s = args.scale.value4<kOut == 2>(p.s[h]);
        v[0] *= s.x; v[1] *= s.y; v[2] *= s.z; v[3] *= s.w;
      }
      if (args.resid != nullptr) {
        v[0] += p.a[h].x; v[1] += p.a[h].y; v[2] += p.a[h].z; v[3] += p.a[h].w;
      }
      if constexpr (kOut == 2) {
        *reinterpret_cast<float4*>(static_cast<float*>(args.y) + at + 32 * h) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
        using T16 = typename std::conditional<kOut == 1, __half, __nv_bfloat16>::type;
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(args.y) + at + 32 * h) =
            make_uint2(Pack16<T16>::pack(v[0], v[1]), Pack16<T16>::pack(v[2], v[3]));
      }
    }
  }
}

}  // namespace fm
