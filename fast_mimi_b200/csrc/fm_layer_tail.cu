// The second half of a transformer layer of few rows in one kernel (sm_100a):
//
//   x1 = x + attn_scale * (core W_o^T)                 y = x1 + mlp_scale * (gelu(LayerNorm(x1) W_1^T) W_2^T)
//
// with 512 channels and an MLP of 2048 (reference: MimiTransformerLayer.forward, src/fast_mimi/model.py:2026-2061).
//
// Latency-bound.  As three kernels (o_proj, LayerNorm + fc1 + GELU, fc2) each pays a launch (3.3 us on the host), a kernel boundary,
// a first load and a reduction over the blocks that share K, for half a microsecond of products.  Here a cluster of 16 blocks
// takes up to 24 rows through all of it: block r owns 32 channels of x1 and y and 128 of the MLP's hidden units, i.e. 288 KB of
// weights, all of it asked for before the wait for the kernel in front: W_o in registers, as the fragments that mma.sync wants (K is
// permuted alike in both operands, so that a lane's share of 32 values of a row is one 16-byte load), W_1 by way of shared
// memory in tensor memory (256 columns, the A operand of fc1), W_2 in shared memory where W_1 lay.  The rows cross the cluster
// twice, as one bulk copy per pair of blocks, counted where it arrives:
//   x1    behind o_proj, since LayerNorm wants whole rows; every block normalises all of them
//   y     partial sums of a block's 128 hidden units, added in the order of the blocks by the owner of 32 channels
// (hidden units would be 2048 x 2 bytes a row to every block, partial sums are 512 x 4).
//
// GPU time of eight FP32 layers, three kernels (for streams two: o_proj behind the attention) -> this one: a clip of 17 frames
// 169 -> 98 us, 64 frames 170 -> 130, 112 frames 187 -> 146, 125 frames 190 -> 161, 168 frames 227 -> 172; 64 streams of two frames 227 -> 200.
// From the wait to the last block's end, us: 8 rows a cluster 4.4 (x1 1.1, LayerNorm 0.7, fc1 with GELU 0.6, fc2 1.1, y 0.7), 16 rows 6.2,
// 24 rows 9: what grows is the two crossings, 2 KB a row into and out of every block at 16 to 19 bytes a cycle (one row instead of eight:
// one stream 80 -> 72 us).  fc1 and fc2 are tcgen05 products with weights as their 128 rows, 32 each, 19 cycles with A in tensor memory and 51
// with A in shared memory, whatever the columns; on mma.sync they took 16 cycles an instruction and scheduler, 1024 per eight rows and
// product (8, 16, 24 rows: 4.9, 8, 12 us).
#include <type_traits>

#include "fm_common.cuh"
#include "fm_device_fact.h"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_warp_mma.cuh"

namespace fm {

namespace tail {
constexpr int kCtas = 16, kHidden = 512, kFfn = 2048;
constexpr int kWarps = 16, kThreads = kWarps * 32, kGroup = 8;     // the first kGroup warps have x1 and y, the others see to W_1 and W_2
constexpr int kCols = kHidden / kCtas;               // 32 channels of x1 and y
constexpr int kUnits = kFfn / kCtas;                 // 128 hidden units
constexpr int kChunks = kHidden / 64;
constexpr int kWBox = 128 * 128;                      // 128 rows of a weight, 64 of K
constexpr int kWBytes = kUnits * kHidden * 2;         // of W_1 and of W_2, one after the other in the same place
constexpr int kTmemCols = 512;                       // W_1 | fc1, two accumulators | fc2
constexpr int kTmemFc1 = kHidden / 2, kTmemFc2 = kTmemFc1 + 2 * 32;
struct Ctl {
  uint64_t w1_full;
  uint64_t w2_full;
  uint64_t x1_full;
  uint64_t y_full;
  uint64_t fc_full[2];                               // fc1's and fc2's products are complete
  uint32_t tmem_base;
  CtaCtl ctl;
};
// W_1, then W_2, then the partial sums of y on their way out | x1, later the partial sums of y, both as they come: [block][row][32
// channels] in FP32 | o_proj's partial sums, later LayerNorm's result and the hidden units | LayerNorm's weights and biases
constexpr int kRowBytes = kHidden * 4, kOperandBytes = kHidden * 2 + kUnits * 2;
static_assert(kGroup * kCols * 4 <= kOperandBytes, "operands and o_proj's partial sums share memory");
constexpr int smem_bytes(int rows) { return 1024 + kWBytes + rows * (kRowBytes + kOperandBytes) + 2 * kHidden * 4 + static_cast<int>(sizeof(Ctl)); }
static_assert(smem_bytes(24) <= 232448, "exceeds the 227 KB a block may use");

// FP32 [row][32 columns] pieces written as fragments (columns lane / 4 .., rows 2 (lane % 4) ..) without bank conflicts
__device__ __forceinline__ int swizzled(int row, int col) { return col ^ (((row >> 1) & 3) << 3); }
// Weights: read before the wait for the kernel in front, and not to be moved behind it.
__device__ __forceinline__ uint4 load_weight(const uint16_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// From this block's shared memory to the same or another place in that of a block of the cluster, counted on its barrier.
__device__ __forceinline__ void copy_to_cta(uint32_t src, uint32_t dst, uint32_t bytes, uint64_t* bar, uint32_t cta) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(map_to_cta(dst, cta)), "r"(src), "r"(bytes), "r"(map_to_cta(smem_u32(bar), cta)) : "memory");
}
// A value of the residual stream as it is stored: type 0 BF16, 1 FP16, 2 FP32.
__device__ __forceinline__ float stream_load(const void* p, long long at, int type) {
  if (type == 2) return __ldcg(static_cast<const float*>(p) + at);
  const uint16_t u = __ldcg(static_cast<const uint16_t*>(p) + at);
  return type == 1 ? __half2float(__ushort_as_half(u)) : __bfloat162float(__ushort_as_bfloat16(u));
}
__device__ __forceinline__ float stream_round(float v, int type) {
  return type == 2 ? v : type == 1 ? __half2float(__float2half_rn(v)) : __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ void stream_store(void* p, long long at, float v, int type) {
  if (type == 2) static_cast<float*>(p)[at] = v;
  else static_cast<uint16_t*>(p)[at] = type == 1 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
}  // namespace tail

struct TailArgs {
  const uint16_t *core, *w_o;            // [M, 512], [512, 512]
  const void* x;                         // [M, 512] of stream_type
  void* y;
  ParamVec attn_scale, mlp_scale, ln_weight, ln_bias;
  float eps;
  int M, rows;                           // rows of a cluster: at most kRows
  int stream_type;
};

// VT: type of core and W_o; TOp: of the MLP's operands
template <typename VT, typename TOp, int kRows>
__global__ void __launch_bounds__(tail::kThreads, 1)
layer_tail_kernel(const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2, const __grid_constant__ TailArgs a, uint32_t idesc, int* status) {
  using namespace tail;
  constexpr int kTiles = kRows / 8;                                            // columns of an mma.sync product: eight rows each
  constexpr int kElems = kRows / kGroup;                                       // of x1 and y, a thread of the first group
  constexpr int kSlice = kRows * kCols * 4;                                    // bytes of a block's channels, at most
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_w = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_x = smem_w + kWBytes;
  uint8_t* smem_h = smem_x + kRows * kRowBytes;
  uint8_t* smem_g = smem_h + kRows * kHidden * 2;
  float* red = reinterpret_cast<float*>(smem_h);
  float4* norm = reinterpret_cast<float4*>(smem_h + kRows * kOperandBytes);
  Ctl* c = reinterpret_cast<Ctl*>(norm + 2 * kHidden / 4);
  CtaCtl* ctl = &c->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = static_cast<int>(threadIdx.x);
  const int g = lane >> 2, q = lane & 3;
  const int rank = static_cast<int>(cluster_cta_rank());
  const int m0 = static_cast<int>(blockIdx.x) / kCtas * a.rows;
  const int n = a.M - m0 < a.rows ? a.M - m0 : a.rows;
  const uint32_t slice = static_cast<uint32_t>(a.rows) * (kCols * 4);          // what a block sends another one
  // A status set before this chain began: nothing is stored.  The blocks of a cluster write into one another's memory and stay to the end.
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  if (tid == 0) {
    mbar_init(&c->w1_full, 1);
    mbar_init(&c->w2_full, 1);
    mbar_init(&c->x1_full, 2 + kThreads - kGroup * 32);       // the other blocks' rows, its own, LayerNorm's parameters
    mbar_init(&c->y_full, 1);
    mbar_init(&c->fc_full[0], 1);
    mbar_init(&c->fc_full[1], 1);
    ctl->abort = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&c->x1_full, (kCtas - 1) * slice);
    mbar_arrive_expect_tx(&c->y_full, kCtas * slice);
    mbar_arrive_expect_tx(&c->w1_full, kWBytes);
#pragma unroll
    for (int kc = 0; kc < kChunks; ++kc) tma_load_2d(smem_w + kc * kWBox, &tmap_w1, &c->w1_full, kc * 64, rank * kUnits);
  }
  if (warp == 1) {
    tmem_alloc(&c->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  cluster_arrive_relaxed();                // this block's memory may be written (its barriers are visible; a release took 1.1 us)
  griddep_launch();
  const uint32_t tmem_base = c->tmem_base, t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  float x1[kElems], mlp_scale = 1.f;       // of the first group: element tid + 256 i, row / 32, channel % 32
  if (warp < kGroup) {
    // ---- x1: all 32 channels of every row, K of this warp's 64, then the sum over the warps
    uint4 w_o[2][2][2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          w_o[mt][j][e] = load_weight(a.w_o + static_cast<size_t>(rank * kCols + mt * 16 + e * 8 + g) * kHidden + warp * 64 + j * 32 + q * 8);
      }
    }
    const float attn_scale = a.attn_scale.data != nullptr ? a.attn_scale.at(rank * kCols + lane) : 1.f;
    if (a.mlp_scale.data != nullptr) mlp_scale = a.mlp_scale.at(rank * kCols + lane);
    griddep_wait();
    uint4 b[kTiles][2];
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      const int row = t * 8 + g;
#pragma unroll
      for (int j = 0; j < 2; ++j)
        b[t][j] = row < n ? __ldcg(reinterpret_cast<const uint4*>(a.core + static_cast<size_t>(m0 + row) * kHidden + warp * 64 + j * 32 + q * 8))
                          : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < kElems; ++i) {
      const int row = (tid >> 5) + i * kGroup;
      x1[i] = row < n ? stream_load(a.x, static_cast<long long>(m0 + row) * kHidden + rank * kCols + lane, a.stream_type) : 0.f;
    }
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      float d[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        d[mt][0] = d[mt][1] = d[mt][2] = d[mt][3] = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_16x8x32<VT>(d[mt], w_o[mt][j][0], w_o[mt][j][1], b[t][j]);
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = t * 8 + 2 * q + (e & 1);
          red[(warp * kRows + row) * kCols + swizzled(row, mt * 16 + g + 8 * (e >> 1))] = d[mt][e];
        }
      }
    }
    named_bar_sync(1, kGroup * 32);
    float* x_out = reinterpret_cast<float*>(smem_x + rank * kSlice);         // this block's own place among the rows is where they start from
#pragma unroll
    for (int i = 0; i < kElems; ++i) {
      const int row = (tid >> 5) + i * kGroup;
      if (row >= a.rows) continue;
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < kGroup; ++w) sum += red[(w * kRows + row) * kCols + swizzled(row, lane)];
      x1[i] = stream_round(x1[i] + attn_scale * sum, a.stream_type);
      x_out[row * kCols + lane] = x1[i];
    }
    fence_proxy_async_smem();
    cluster_wait();                        // every block of the cluster runs
    named_bar_sync(1, kGroup * 32);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < kCtas / kGroup; ++i) {
        const int to = warp + i * kGroup;
        if (to == rank) mbar_arrive(&c->x1_full);
        else copy_to_cta(smem_u32(x_out), smem_u32(x_out), slice, &c->x1_full, static_cast<uint32_t>(to));
      }
    }
    __syncwarp();
  } else {
    // ---- meanwhile, or ahead of all that: W_1 into tensor memory (hidden unit 32 (warp % 4) + lane, two values of K a column), then W_2
    // into its place.  Not by all warps ahead of the wait: a cluster that starts late would wait for it, as one in six or seven
    // does (a GPC has few SMs more than a cluster, and the attention's blocks sit on some).  (Loaded from global memory by the lane
    // that stores it, a line a lane, it took 4 us.)
    {
      const int i = tid - kGroup * 32;     // LayerNorm's weights and biases, four a thread
      norm[i] = i < kHidden / 4 ? a.ln_weight.load4(4 * i) : a.ln_bias.load4(4 * i - kHidden);
    }
    mbar_wait(&c->w1_full, 0, ctl, status, kErrWaitTma);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kChunks / 2; ++i) {
      const int kc = ((warp >> 2) & 1) * (kChunks / 2) + i;
      uint32_t r[32];
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const uint4 v = *reinterpret_cast<const uint4*>(smem_w + kc * kWBox + sw128_offset((warp & 3) * 32 + lane, p));
        r[4 * p] = v.x; r[4 * p + 1] = v.y; r[4 * p + 2] = v.z; r[4 * p + 3] = v.w;
      }
      tmem_st32(t_row + kc * 32, r);
    }
    tmem_st_wait();
    tc_fence_before_sync();                // the products follow behind a barrier of the block
    fence_proxy_async_smem();
    named_bar_sync(2, (kWarps - kGroup) * 32);
    if (warp == kGroup && lane == 0) {
      mbar_arrive_expect_tx(&c->w2_full, kWBytes);
#pragma unroll
      for (int i = 0; i < kWBytes / kWBox; ++i)        // 128 channels, half of the hidden units
        tma_load_2d(smem_w + i * kWBox, &tmap_w2, &c->w2_full, rank * kUnits + (i & 1) * 64, (i >> 1) * 128);
    }
    __syncwarp();
    cluster_wait();                        // with the first group's
    mbar_arrive(&c->x1_full);              // LayerNorm's parameters are there
  }

  // ---- LayerNorm, one warp a row, the same sums in the same order as layernorm512_kernel
  mbar_wait_cluster(&c->x1_full, 0, ctl, status, kErrWaitConsumer);
  __syncwarp();
  {
    constexpr int kMine = (kRows + kWarps - 1) / kWarps;
    float v[kMine][4][4], sum[kMine], sq[kMine];
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int row = warp + kWarps * i < a.rows ? warp + kWarps * i : 0;
      sum[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {        // channels 128 j + 4 lane ..: block 4 j + lane / 8
        const float4 u = *reinterpret_cast<const float4*>(smem_x + (4 * j + (lane >> 3)) * kSlice + row * (kCols * 4) + (lane & 7) * 16);
        v[i][j][0] = u.x; v[i][j][1] = u.y; v[i][j][2] = u.z; v[i][j][3] = u.w;
        sum[i] += (u.x + u.y) + (u.z + u.w);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < kMine; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
    }
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const float mean = sum[i] * (1.0f / kHidden);
      sq[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[i][j][e] -= mean;
          sq[i] += v[i][j][e] * v[i][j][e];
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < kMine; ++i) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
    }
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int row = warp + kWarps * i;
      if (row < a.rows) {
        const float rstd = rsqrtf(sq[i] * (1.0f / kHidden) + a.eps);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 wf = norm[32 * j + lane], bf = norm[128 + 32 * j + lane];
          const float* x = v[i][j];
          // chunk 2 j + lane / 16, 16-byte piece (lane % 16) / 2, its lower or upper half
          *reinterpret_cast<uint2*>(smem_h + (2 * j + (lane >> 4)) * (kRows * 128) + sw128_offset(row, (lane & 15) >> 1) + (lane & 1) * 8) =
              make_uint2(Pack16<TOp>::pack(x[0] * rstd * wf.x + bf.x, x[1] * rstd * wf.y + bf.y),
                         Pack16<TOp>::pack(x[2] * rstd * wf.z + bf.z, x[3] * rstd * wf.w + bf.w));
        }
      }
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  cluster_arrive_relaxed();                // x1 has been read: partial sums of y may come

  // ---- fc1: 128 hidden units as rows of the product, 256 of K in each of two accumulators (fm_ln_linear.cu).  Columns past kRows (N is a
  // multiple of 16) are what lies behind the operand.
  if (warp == 0) {
    tc_fence_after_sync();
    const uint64_t h = umma_desc_sw128(smem_u32(smem_h));
    const bool one = elect_one();
    for (int kc = 0; kc < kChunks; ++kc) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (one)
          tc_mma_ts(tmem_base + kTmemFc1 + kc / (kChunks / 2) * 32, tmem_base + kc * 32 + ks * 8, h + static_cast<uint64_t>(kc * kRows * 128 >> 4) + 2u * ks,
                    idesc, (kc % (kChunks / 2) | ks) != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&c->fc_full[0]);
    __syncwarp();
  }
  mbar_wait(&c->fc_full[0], 0, ctl, status, kErrWaitMma);
  __syncwarp();
  tc_fence_after_sync();
  {
    // hidden unit 32 (warp % 4) + lane, a few rows a warp
    constexpr int kN = kRows == 24 ? 8 : 4;
    const int row0 = (warp >> 2) * kN, unit = (warp & 3) * 32 + lane;
    if (row0 < kRows) {
      uint32_t u[kN], w[kN];
      if constexpr (kN == 8) {
        tmem_ld8(t_row + kTmemFc1 + row0, u);
        tmem_ld8(t_row + kTmemFc1 + 32 + row0, w);
      } else {
        tmem_ld4(t_row + kTmemFc1 + row0, u);
        tmem_ld4(t_row + kTmemFc1 + 32 + row0, w);
      }
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kN; i += 2) {
        float v0 = __uint_as_float(u[i]) + __uint_as_float(w[i]), v1 = __uint_as_float(u[i + 1]) + __uint_as_float(w[i + 1]);
        gelu_erf2(v0, v1);
        const uint32_t p = Pack16<TOp>::pack(v0, v1);
        uint8_t* chunk = smem_g + (unit >> 6) * (kRows * 128) + (unit & 7) * 2;
        *reinterpret_cast<uint16_t*>(chunk + sw128_offset(row0 + i, (unit & 63) >> 3)) = static_cast<uint16_t>(p);
        *reinterpret_cast<uint16_t*>(chunk + sw128_offset(row0 + i + 1, (unit & 63) >> 3)) = static_cast<uint16_t>(p >> 16);
      }
    }
    tc_fence_before_sync();
    fence_proxy_async_smem();
  }
  if (warp == 0) mbar_wait(&c->w2_full, 0, ctl, status, kErrWaitTma);      // here: right behind a wait products issue at half the rate
  __syncthreads();

  // ---- fc2: partial sums of all 512 channels, 128 a product; a warp has those of block `warp`, staged where W_1 lay
  if (warp == 0) {
    tc_fence_after_sync();
    const uint64_t w2 = umma_desc_sw128(smem_u32(smem_w)), hidden = umma_desc_sw128(smem_u32(smem_g));
    const bool one = elect_one();
    for (int t = 0; t < kHidden / 128; ++t) {
#pragma unroll
      for (int ks = 0; ks < kUnits / 16; ++ks)
        if (one)
          tc_mma_ss(tmem_base + kTmemFc2 + t * 32, w2 + static_cast<uint64_t>((2 * t + (ks >> 2)) * kWBox >> 4) + 2u * (ks & 3),
                    hidden + static_cast<uint64_t>((ks >> 2) * kRows * 128 >> 4) + 2u * (ks & 3), idesc, ks != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&c->fc_full[1]);
    __syncwarp();
  }
  mbar_wait(&c->fc_full[1], 0, ctl, status, kErrWaitMma);
  __syncwarp();
  tc_fence_after_sync();
  float* stage = reinterpret_cast<float*>(smem_w + warp * kSlice);
#pragma unroll
  for (int r0 = 0; r0 < kRows; r0 += 8) {
    uint32_t u[8];
    tmem_ld8(t_row + kTmemFc2 + (warp >> 2) * 32 + r0, u);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i) stage[(r0 + i) * kCols + lane] = __uint_as_float(u[i]);
  }
  tc_fence_before_sync();
  fence_proxy_async_smem();
  __syncwarp();
  cluster_wait();                          // no block reads x1 any more
  if (lane == 0) copy_to_cta(smem_u32(stage), smem_u32(smem_x + rank * kSlice), slice, &c->y_full, static_cast<uint32_t>(warp));
  __syncwarp();
  mbar_wait_cluster(&c->y_full, 0, ctl, status, kErrWaitConsumer);
  __syncwarp();
  cluster_arrive_relaxed();                // this block's rows are complete; see the end
  if (warp < kGroup) {
#pragma unroll
    for (int i = 0; i < kElems; ++i) {
      const int row = (tid >> 5) + i * kGroup;
      if (row < n) {
        float sum = 0.f;
#pragma unroll
        for (int s = 0; s < kCtas; ++s) sum += *reinterpret_cast<const float*>(smem_x + s * kSlice + (row * kCols + lane) * 4);
        if (!skip) stream_store(a.y, static_cast<long long>(m0 + row) * kHidden + rank * kCols + lane, x1[i] + mlp_scale * sum, a.stream_type);
      }
    }
  }
  cluster_wait();                          // every block has its rows: nobody's copies still read this block's memory
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);      // copies that may still be in flight get time to land
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

namespace {
template <typename Kern>
bool allow(Kern kern, int bytes) {
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), bytes) == 0 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
    return true;
  (void)cudaGetLastError();
  return false;
}

// Clusters that the device runs at once; 0: none, or not to be found out just now.  Asked of one kernel for all: it allows every
// one of them its clusters, and none takes more than the largest.
template <typename VT, typename TOp>
bool allow_rows() {
  using namespace tail;
  return allow(layer_tail_kernel<VT, TOp, 8>, smem_bytes(8)) && allow(layer_tail_kernel<VT, TOp, 16>, smem_bytes(16)) &&
         allow(layer_tail_kernel<VT, TOp, 24>, smem_bytes(24));
}

int tail_clusters() {
  using namespace tail;
  static DeviceFact clusters;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const int n = clusters.get(dev, [] {
    if (!allow_rows<__half, __half>() || !allow_rows<__half, __nv_bfloat16>() || !allow_rows<__nv_bfloat16, __half>() ||
        !allow_rows<__nv_bfloat16, __nv_bfloat16>())
      return -1;
    return resident_clusters(layer_tail_kernel<__half, __half, 24>, kThreads, smem_bytes(24), kCtas);
  });
  return n > 0 ? n : 0;
}

// Rows of a cluster for M rows in one wave, 0 where 24 are too few (7 clusters on a B200: 168 rows in all).  Products are made for 8,
// 16 or 24 rows: as few as the clusters that the device holds can do with.  Fewer rows than that cost every block less in its crossings, so
// they are dealt evenly to five clusters at least: a sixth or seventh often finds no GPC with 16 free SMs until the kernel in front ends
// (eight layers of a clip of 17 frames: 98 us on five, 102 on six, 107 on two; 40 streams 140 on five, 146 on six).  Where each block of the kernel in
// front has an SM to itself (`beside` of them), to as many as the others hold, but three (12 streams beside 96 blocks 87 us on
// three, 99 on four, 103 on one; 18 beside 144 109 on three, 111 on five, 142 on one).
int rows_of_cluster(int M, int beside) {
  const int held = tail_clusters();
  int tile = 8;
  while (tile < 24 && M > tile * held) tile += 8;
  if (M > tile * held) return 0;
  int clusters = held < 5 ? held : 5;
  if (beside > 0) {
    const int room = (sm_count() - beside) / tail::kCtas;
    if (room < clusters) clusters = room < 3 ? 3 : room;
  }
  const int least = (M + tile - 1) / tile;
  if (clusters < least) clusters = least;
  return (M + clusters - 1) / clusters;
}

template <typename VT, typename TOp>
int launch_rows(int rows, const CUtensorMap& tmap_w1, const CUtensorMap& tmap_w2, const TailArgs& a, int* status, cudaStream_t st, int dependent) {
  using namespace tail;
  const int tile = (rows + 7) / 8 * 8;
  auto kern = tile == 8 ? layer_tail_kernel<VT, TOp, 8> : tile == 16 ? layer_tail_kernel<VT, TOp, 16> : layer_tail_kernel<VT, TOp, 24>;
  const int fmt = std::is_same<TOp, __half>::value ? 0 : 1;
  const uint32_t idesc = umma_idesc_f16(128, tile <= 16 ? 16 : 32, fmt, fmt, 0, 0);
  return launch_kernel(kern, dim3(kCtas * ((a.M + rows - 1) / rows)), kThreads, smem_bytes(tile), st, kCtas, dependent, tmap_w1, tmap_w2, a, idesc, status);
}
}  // namespace

bool layer_tail_takes(int M, int ffn) { return ffn == tail::kFfn && M > 0 && rows_of_cluster(M, 0) > 0; }

int launch_layer_tail(const LayerTail& t, int M, int* status, cudaStream_t st, int dependent) {
  const int rows = M > 0 ? rows_of_cluster(M, t.beside) : 0;
  if (rows == 0 || t.stream_type < 0 || t.stream_type > 2) return -1;
  if ((reinterpret_cast<uintptr_t>(t.core) | reinterpret_cast<uintptr_t>(t.x) | reinterpret_cast<uintptr_t>(t.y) |
       reinterpret_cast<uintptr_t>(t.w_o) | reinterpret_cast<uintptr_t>(t.w_fc1) | reinterpret_cast<uintptr_t>(t.w_fc2) |
       reinterpret_cast<uintptr_t>(t.attn_scale.data) | reinterpret_cast<uintptr_t>(t.mlp_scale.data) |
       reinterpret_cast<uintptr_t>(t.ln_weight.data) | reinterpret_cast<uintptr_t>(t.ln_bias.data)) & 15u)
    return -3;
  CUtensorMap tmap_w1, tmap_w2;
  int rc = encode_rows_16bit(&tmap_w1, t.w_fc1, tail::kFfn, tail::kHidden, tail::kUnits, 64);
  if (rc == 0) rc = encode_rows_16bit(&tmap_w2, t.w_fc2, tail::kHidden, tail::kFfn, 128, 64);
  if (rc != 0) return rc;
  const TailArgs a = {static_cast<const uint16_t*>(t.core), static_cast<const uint16_t*>(t.w_o), t.x, t.y,
                      t.attn_scale, t.mlp_scale, t.ln_weight, t.ln_bias, t.eps, M, rows, t.stream_type};
  if (t.value_fp16)
    return t.tc_fp16 ? launch_rows<__half, __half>(rows, tmap_w1, tmap_w2, a, status, st, dependent)
                     : launch_rows<__half, __nv_bfloat16>(rows, tmap_w1, tmap_w2, a, status, st, dependent);
  return t.tc_fp16 ? launch_rows<__nv_bfloat16, __half>(rows, tmap_w1, tmap_w2, a, status, st, dependent)
                   : launch_rows<__nv_bfloat16, __nv_bfloat16>(rows, tmap_w1, tmap_w2, a, status, st, dependent);
}

}  // namespace fm
