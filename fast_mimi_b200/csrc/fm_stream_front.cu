// The first half of a layer's call for a few live streams in one kernel (sm_100a): T <= 8 new frames per stream at positions past ..
//
//   q | k | v = LayerNorm(x) W_qkv^T, RoPE       core = attention over the stream's ring and the new rows       ring <- new k, v
//
// (reference: MimiTransformerLayer.forward, src/fast_mimi/model.py:2026-2058, with MimiAttention.forward and MimiKVCache.update,
// :1897-1912, :450-471).  What it does between q, k, v and core is fm_stream_attn.cu's, for one item a block.
//
// Latency-bound: as two kernels (fm_ln_linear.cu, fm_stream_attn.cu) the host pays a launch more (3.3 us of 14 a layer), the GPU a kernel
// boundary and the way of q, k and v through memory, each of which waits for a first load.  Here a block has one head of one
// stream: 192 rows of W_qkv, 192 KB, on the chip before the wait for the kernel in front.  k and v's are the A operand of a tcgen05 product,
// by way of shared memory in tensor memory (256 columns; 19 cycles an instruction): the ring's new rows have the bits that the other
// projection kernels of a layer's call give them, K = 512 in one accumulator.  q's are in registers, as the fragments that mma.sync wants (K permuted alike in both operands, so that
// a lane's share of 32 values of a row is one 16-byte load), a quarter of K a warp: both go on at once.  (All three on mma.sync took 1.2 us
// at 16 cycles an instruction and scheduler.)  The ring's rows (64 KB) come while that runs: not ahead of the wait, since the kernel that
// opens a chain cannot know what wrote them.  Then 16 slots of the ring a warp.
//
// Eight layers, two kernels -> this one, GPU time in a captured graph (and called eagerly, where the host's launches are the limit), us:
// 1 FP32 stream of one frame 98 -> 80 (123 -> 103), 12 streams 118 -> 92, 18 streams 122 -> 110, 5 of eight frames 129 -> 96 (133 -> 103), 18 of
// eight 180 -> 164; BF16 alike.  From the wait to the end 3.9 us: LayerNorm 1.0, projection 0.8, q, k and v in place 0.3, scores 0.6,
// probabilities and products with V 0.65, the sixteen warps' results as one 0.5.
#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_stream_math.cuh"
#include "fm_warp_mma.cuh"

namespace fm {

namespace front {
constexpr int kWarps = 16, kThreads = kWarps * 32, kMaxT = 8;
constexpr int kHidden = 512, kGroups = 4, kShare = kHidden / kGroups;      // K in four groups of warps
constexpr int kTileBytes = 256 * 128;                 // K or V of the ring, padded to 256 slots
constexpr int kWBox = 64 * 128, kWBytes = 16 * kWBox; // 64 rows, 64 of K; k's and v's rows of a head
constexpr int kNewBytes = 16 * 128;                   // new K or V rows, padded to 16
constexpr int kQRow = 72;                             // values of a row of q, padded
constexpr int kHBytes = 9 * 1024;                     // LayerNorm's result, eight chunks of 64 channels; the product reads 16 rows
constexpr int kTmemCols = 512, kTmemD = kHidden / 2;  // W_k and W_v | k and v
struct Shared {
  uint64_t w_full;
  uint64_t kv_full;
  uint64_t ring_full;
  uint32_t tmem_base;
  CtaCtl ctl;
  float m[kWarps][kMaxT];
  float l[kWarps][kMaxT];
  float q_part[kGroups][kMaxT][64];                   // partial sums of q
  float kv[kMaxT][128];
  alignas(16) uint16_t q[kMaxT * kQRow];
};
static_assert(sizeof(Shared) % 16 == 0 && kQRow % 8 == 0, "read in pieces of 16 bytes");
// Ring | results of the warps | LayerNorm's result | new rows.  The weights pass through the first two on their way.
constexpr int kMergeBytes = kWarps * kMaxT * 64 * 4;
constexpr int kPassBytes = 2 * kTileBytes + kMergeBytes > kWBytes ? 2 * kTileBytes + kMergeBytes : kWBytes;
constexpr int kSmemBytes = 1024 + kPassBytes + kHBytes + 2 * kNewBytes + static_cast<int>(sizeof(Shared));
static_assert(kSmemBytes <= 232448, "exceeds the 227 KB a block may use");

// A column of 16 or more under rows as fragments have them (columns lane / 4 .., rows 2 (lane % 4) ..), without bank conflicts
__device__ __forceinline__ int swizzled(int row, int col) { return col ^ (((row >> 1) & 3) << 3); }
__device__ __forceinline__ uint4 load_weight(const uint16_t* p) {      // not to be moved behind the wait
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
}  // namespace front

struct FrontArgs {
  const void* x;                 // [S, T, 512] of stream_type
  ParamVec ln_weight, ln_bias;
  const uint16_t* w_qkv;         // [1536, 512]
  const float *cos, *sin;
  long long cos_bstride;
  uint16_t *ring_k, *ring_v;     // [S, 8, slots, 64]
  uint16_t* core;                // [S, T, 512]
  float eps, scale_log2e;
  int stream_type, T, delta, slots, window;
  int first, next;               // slots of the oldest visible row and of the first new one
  int n_loaded;                  // ring rows that the tensor maps' boxes cover: min(past, slots)
};

// VT: type of the ring's values, v and core; TOp: of the projection's operands
template <typename VT, typename TOp>
__global__ void __launch_bounds__(front::kThreads, 1)
stream_front_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_w,
                    const __grid_constant__ FrontArgs a, uint32_t idesc, int* status) {
  using namespace front;
  if (chain_stopped(status)) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tile_k = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tile_v = tile_k + kTileBytes;
  float (*merge)[kMaxT][64] = reinterpret_cast<float (*)[kMaxT][64]>(tile_v + kTileBytes);
  uint8_t* smem_h = tile_k + kPassBytes;
  uint8_t* new_k = smem_h + kHBytes;
  uint8_t* new_v = new_k + kNewBytes;
  Shared* c = reinterpret_cast<Shared*>(new_v + kNewBytes);
  CtaCtl* ctl = &c->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = static_cast<int>(threadIdx.x);
  const int g = lane >> 2, q = lane & 3;
  const int s = static_cast<int>(blockIdx.x) >> 3, h = static_cast<int>(blockIdx.x) & 7;
  const int kg = warp & 3, og = warp >> 2;             // q: quarter of K, 16 of the 64 rows
  if (tid == 0) {
    mbar_init(&c->w_full, 1);
    mbar_init(&c->kv_full, 1);
    mbar_init(&c->ring_full, 1);
    ctl->abort = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&c->w_full, kWBytes);
#pragma unroll
    for (int kc = 0; kc < 8; ++kc) {
      tma_load_2d(tile_k + 2 * kc * kWBox, &tmap_w, &c->w_full, kc * 64, kHidden + h * 64);
      tma_load_2d(tile_k + (2 * kc + 1) * kWBox, &tmap_w, &c->w_full, kc * 64, 2 * kHidden + h * 64);
    }
  }
  if (warp == 1) {
    tmem_alloc(&c->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  uint4 w[4][2];
  {
    const uint16_t* row = a.w_qkv + static_cast<size_t>(h * 64 + og * 16 + g) * kHidden + kg * kShare + q * 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w[j][0] = load_weight(row + j * 32);
      w[j][1] = load_weight(row + 8 * kHidden + j * 32);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = c->tmem_base, t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  // W_k and W_v into tensor memory: rows 0 .. 63 and 64 .. 127 of the product, two values of K a column
  mbar_wait(&c->w_full, 0, ctl, status, kErrWaitTma);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int kc = 2 * og + i;
    uint32_t r[32];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const uint4 v = *reinterpret_cast<const uint4*>(tile_k + 2 * kc * kWBox + sw128_offset((warp & 3) * 32 + lane, p));
      r[4 * p] = v.x; r[4 * p + 1] = v.y; r[4 * p + 2] = v.z; r[4 * p + 3] = v.w;
    }
    tmem_st32(t_row + kc * 32, r);
  }
  tmem_st_wait();
  tc_fence_before_sync();                              // the product follows behind a barrier of the block
  __syncthreads();
  // Slots past the loaded ones and rows past the new ones are never written: zeros, so that a probability of zero times
  // what lies there is zero.
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < 2 * (256 - a.n_loaded) * 8; i += kThreads) {
    const int per = (256 - a.n_loaded) * 8, tile = i / per, piece = i % per;
    *reinterpret_cast<uint4*>(tile_k + tile * kTileBytes + a.n_loaded * 128 + piece * 16) = zero;
  }
  if (tid < 2 * kNewBytes / 16) *reinterpret_cast<uint4*>(new_k + tid * 16) = zero;
  for (int i = tid; i < kMaxT * kQRow / 8; i += kThreads) *reinterpret_cast<uint4*>(c->q + i * 8) = zero;
  fence_proxy_async_smem();
  __syncthreads();
  griddep_wait();
  griddep_launch();                        // this kernel opens the chain
  if (tid == 0 && a.n_loaded > 0) {
    mbar_arrive_expect_tx(&c->ring_full, 2u * static_cast<uint32_t>(a.n_loaded) * 128u);
    tma_load_2d(tile_k, &tmap_k, &c->ring_full, 0, static_cast<int>(blockIdx.x) * a.slots);
    tma_load_2d(tile_v, &tmap_v, &c->ring_full, 0, static_cast<int>(blockIdx.x) * a.slots);
  }

  // ---- LayerNorm, one warp a row, the same sums in the same order as layernorm512_kernel.  (In the fragments' own layout, four warps
  // each with the same quarter of all rows, it took 0.9 us.)
  const int t_rope = warp & 7;             // row (of eight) and dimension lane of q or k that this thread turns below
  float cosv = 0.f, sinv = 0.f;
  if (warp < a.T) {
    float v[4][4];
    uint4 nw[4], nb[4];
    const long long at = (static_cast<long long>(s) * a.T + warp) * kHidden + 4 * lane;
    if (a.stream_type == 2) {
#pragma unroll
      for (int j = 0; j < 4; ++j) load4<2>(a.x, at + 128 * j, v[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        nw[j] = a.ln_weight.raw4<true>(128 * j + 4 * lane);
        nb[j] = a.ln_bias.raw4<true>(128 * j + 4 * lane);
      }
    } else {
      uint2 u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = __ldcg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(a.x) + at + 128 * j));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        nw[j] = a.ln_weight.raw4(128 * j + 4 * lane);
        nb[j] = a.ln_bias.raw4(128 * j + 4 * lane);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 lo = a.stream_type == 1 ? Pack16<__half>::unpack(u[j].x) : Pack16<__nv_bfloat16>::unpack(u[j].x);
        const float2 hi = a.stream_type == 1 ? Pack16<__half>::unpack(u[j].y) : Pack16<__nv_bfloat16>::unpack(u[j].y);
        v[j][0] = lo.x; v[j][1] = lo.y; v[j][2] = hi.x; v[j][3] = hi.y;
      }
    }
    float sum = 0.f, sq = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) sum += (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum * (1.0f / kHidden);
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
    const float rstd = rsqrtf(sq * (1.0f / kHidden) + a.eps);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 wf = a.ln_weight.value4(nw[j]), bf = a.ln_bias.value4(nb[j]);
      *reinterpret_cast<uint2*>(smem_h + (2 * j + (lane >> 4)) * 1024 + sw128_offset(warp, (lane & 15) >> 1) + (lane & 1) * 8) =
          make_uint2(Pack16<TOp>::pack(v[j][0] * rstd * wf.x + bf.x, v[j][1] * rstd * wf.y + bf.y),
                     Pack16<TOp>::pack(v[j][2] * rstd * wf.z + bf.z, v[j][3] * rstd * wf.w + bf.w));
    }
  }
  if (t_rope < a.T) {
    const long long at = s * a.cos_bstride + static_cast<long long>(t_rope) * 64 + lane;
    cosv = __ldg(a.cos + at);
    sinv = __ldg(a.sin + at);
  }
  fence_proxy_async_smem();
  __syncthreads();

  // ---- projection: outputs as rows, the frames as columns.  What lies past the new rows stays in columns that nobody reads.
  if (warp == 0) {
    tc_fence_after_sync();
    const uint64_t hd = umma_desc_sw128(smem_u32(smem_h));
    const bool one = elect_one();
    for (int kc = 0; kc < 8; ++kc) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (one)
          tc_mma_ts(tmem_base + kTmemD, tmem_base + kc * 32 + ks * 8, hd + static_cast<uint64_t>(kc * 1024 >> 4) + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&c->kv_full);
    __syncwarp();
  }
  {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 b = *reinterpret_cast<const uint4*>(smem_h + (2 * kg + (j >> 1)) * 1024 + sw128_offset(g, 4 * (j & 1) + q));
      mma_16x8x32<TOp>(d, w[j][0], w[j][1], b);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = 2 * q + (e & 1);
      c->q_part[kg][row][swizzled(row, og * 16 + g + 8 * (e >> 1))] = d[e];
    }
  }
  if (warp < 4) {
    mbar_wait(&c->kv_full, 0, ctl, status, kErrWaitMma);
    __syncwarp();
    tc_fence_after_sync();
    uint32_t r[8];
    tmem_ld8(t_row + kTmemD, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < kMaxT; ++i) c->kv[i][warp * 32 + lane] = __uint_as_float(r[i]);
    tc_fence_before_sync();
  }
  __syncthreads();
  {
    auto cell = [&](uint8_t* tile, int row, int d) { return reinterpret_cast<uint16_t*>(tile + sw128_offset(row, d >> 3) + (d & 7) * 2); };
    const int row = t_rope;                            // warps 0 .. 7: q, 8 .. 15: k
    if (row < a.T) {
      auto total = [&](int d) {
        const int at = swizzled(row, d);
        return (c->q_part[0][row][at] + c->q_part[1][row][at]) + (c->q_part[2][row][at] + c->q_part[3][row][at]);
      };
      const float lo = warp < 8 ? total(lane) : c->kv[row][lane], hi = warp < 8 ? total(32 + lane) : c->kv[row][32 + lane];
      // contracted and rounded as in the other projection kernels, whose rows this kernel's stand beside in a ring
      const uint32_t y = Pack16<__nv_bfloat16>::pack(__fmaf_rn(lo, cosv, -__fmul_rn(hi, sinv)), __fmaf_rn(hi, cosv, __fmul_rn(lo, sinv)));
      if (warp < 8) {
        c->q[row * kQRow + lane] = static_cast<uint16_t>(y);
        c->q[row * kQRow + 32 + lane] = static_cast<uint16_t>(y >> 16);
      } else {
        *cell(new_k, row, lane) = static_cast<uint16_t>(y);
        *cell(new_k, row, 32 + lane) = static_cast<uint16_t>(y >> 16);
      }
    }
    const int v_row = warp >> 1, d = (warp & 1) * 32 + lane;
    if (v_row < a.T) *cell(new_v, v_row, d) = static_cast<uint16_t>(Pack16<VT>::pack(c->kv[v_row][64 + d], 0.f));
  }
  __syncthreads();

  // ---- attention: 16 slots of the ring a warp, the last one the new rows besides
  if (a.n_loaded > 0) mbar_wait(&c->ring_full, 0, ctl, status, kErrWaitTma);
  __syncwarp();
  // The ring's old rows are here: the new ones take their slots (of two rows for one slot the newer stays).
  if (tid < 128) {
    const int piece = tid & 63, t = piece >> 3;
    if (t < a.T && t >= a.T - a.slots) {
      uint16_t* ring = tid < 64 ? a.ring_k : a.ring_v;
      int slot = a.next + t;
      while (slot >= a.slots) slot -= a.slots;
      *reinterpret_cast<uint4*>(ring + (static_cast<size_t>(blockIdx.x) * a.slots + slot) * 64 + (piece & 7) * 8) =
          *reinterpret_cast<const uint4*>((tid < 64 ? new_k : new_v) + sw128_offset(t, piece & 7));
    }
  }
  const int slot0 = warp * 16;
  {
    // What a slot of V holds that is no longer visible to anyone must not reach the sums through 0 * x.
    const int j = slot0 + (lane & 15);
    int r = j - a.first;
    if (r < 0) r += a.slots;
    if (j < a.n_loaded && r >= a.delta) {
#pragma unroll
      for (int p = 0; p < 4; ++p) *reinterpret_cast<uint4*>(tile_v + j * 128 + ((lane >> 4) * 4 + p) * 16) = zero;
    }
    __syncwarp();
  }
  const bool has_ring = a.n_loaded > slot0, has_new = warp == kWarps - 1;
  auto in_use = [&](int mt) { return mt == 0 ? has_ring : has_new; };            // the same for the whole warp
  const int cpair = 2 * q;
  float sc[2][4];                                      // keys g (two queries) and g + 8
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) sc[mt][0] = sc[mt][1] = sc[mt][2] = sc[mt][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(c->q + g * kQRow + ks * 16 + cpair), b1 = *reinterpret_cast<const uint32_t*>(c->q + g * kQRow + ks * 16 + 8 + cpair);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      if (in_use(mt)) {
        uint32_t ka[4];                                // keys lane % 16, dimensions 16 ks + 8 (lane / 16) ..
        ldmatrix4(ka, smem_u32(mt == 0 ? tile_k : new_k) + sw128_offset((mt == 0 ? slot0 : 0) + (lane & 15), 2 * ks + (lane >> 4)));
        mma_16x8x16<__nv_bfloat16>(sc[mt], ka, b0, b1);
      }
    }
  }
  // visible rows of query t: delta + t - window < r <= delta + t
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, m_use[2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int key = g + 8 * (e >> 1), t = cpair + (e & 1);
      int r = a.delta + key;
      if (mt == 0) {
        const int j = slot0 + key;
        r = j - a.first;
        if (r < 0) r += a.slots;
        if (j >= a.n_loaded || r >= a.delta) r = -(1 << 28);
      }
      const bool seen = in_use(mt) && r <= a.delta + t && r > a.delta + t - a.window;
      sc[mt][e] = seen ? sc[mt][e] * a.scale_log2e : -INFINITY;
      m[e & 1] = fmaxf(m[e & 1], sc[mt][e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], x));
    m_use[e] = m[e] == -INFINITY ? 0.f : m[e] - Parts<VT>::kShift;
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sc[mt][e] = ex2_approx(sc[mt][e] - m_use[e & 1]);
      l[e & 1] += sc[mt][e];
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], x);
  }
  // O^T = V^T P^T, dimensions as rows.  A score fragment has keys along the lanes' groups and queries inside them; as an operand it
  // must be the other way round (movmatrix).
  float o[4][4];                                       // dimensions 16 d + g and + 8, two queries each
#pragma unroll
  for (int d = 0; d < 4; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    if (in_use(mt)) {
      uint32_t p0[Parts<VT>::kParts], p1[Parts<VT>::kParts];
      split_pair<VT>(sc[mt][0], sc[mt][1], p0);
      split_pair<VT>(sc[mt][2], sc[mt][3], p1);
#pragma unroll
      for (int i = 0; i < Parts<VT>::kParts; ++i) {
        p0[i] = movmatrix_trans(p0[i]);
        p1[i] = movmatrix_trans(p1[i]);
      }
      const uint32_t base = smem_u32(mt == 0 ? tile_v : new_v);
      const int key = (mt == 0 ? slot0 : 0) + (lane & 7) + ((lane >> 4) << 3);
      uint32_t va[4][4];
#pragma unroll
      for (int d = 0; d < 4; ++d) ldmatrix4_trans(va[d], base + sw128_offset(key, 2 * d + ((lane >> 3) & 1)));
#pragma unroll
      for (int i = 0; i < Parts<VT>::kParts; ++i) {
#pragma unroll
        for (int d = 0; d < 4; ++d) mma_16x8x16<VT>(o[d], va[d], p0[i], p1[i]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = cpair + e;
    if (t < a.T) {
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        merge[warp][t][d * 16 + g] = o[d][e];
        merge[warp][t][d * 16 + 8 + g] = o[d][2 + e];
      }
      if (g == 0) {
        c->m[warp][t] = m[e];
        c->l[warp][t] = l[e];
      }
    }
  }
  __syncthreads();
  const int t = tid >> 6, d = tid & 63;
  if (t < a.T) {
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) mx = fmaxf(mx, c->m[i][t]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const float f = ex2_approx(c->m[i][t] - mx);     // 0 for a warp that saw no row
      num = fmaf(f, merge[i][t][d], num);
      den = fmaf(f, c->l[i][t], den);
    }
    a.core[(static_cast<size_t>(s) * a.T + t) * kHidden + h * 64 + d] = static_cast<uint16_t>(Pack16<VT>::pack(num / den, 0.f));
  }
  if (ctl->abort) __nanosleep(20000);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// While every head of every stream has an SM: a second wave costs as much as the first, and 19 streams take 123 us in two kernels.
bool stream_front_takes(int S, int T, int slots) { return T <= front::kMaxT && slots <= 256 && 8ll * S <= sm_count(); }

int launch_stream_front(const StreamFront& f, int S, int T, int past, int slots, int window, float scale, int* status, cudaStream_t st, int dependent) {
  using namespace front;
  if (S <= 0 || T <= 0 || past < 0 || window <= 0 || slots < window || !stream_front_takes(S, T, slots) || f.stream_type < 0 || f.stream_type > 2) return -1;
  if ((reinterpret_cast<uintptr_t>(f.x) | reinterpret_cast<uintptr_t>(f.ln_weight.data) | reinterpret_cast<uintptr_t>(f.ln_bias.data) |
       reinterpret_cast<uintptr_t>(f.w_qkv) | reinterpret_cast<uintptr_t>(f.ring_k) | reinterpret_cast<uintptr_t>(f.ring_v) |
       reinterpret_cast<uintptr_t>(f.core)) & 15u)
    return -3;
  const int delta = past < window - 1 ? past : window - 1, n_loaded = past < slots ? past : slots;
  CUtensorMap tk = {}, tv = {}, tw;
  int rc = encode_rows_16bit(&tw, f.w_qkv, 1536, kHidden, 64, 64);
  if (rc == 0 && n_loaded > 0) rc = encode_rows_16bit(&tk, f.ring_k, static_cast<uint64_t>(S) * 8 * slots, 64, static_cast<uint32_t>(n_loaded), 64);
  if (rc == 0 && n_loaded > 0) rc = encode_rows_16bit(&tv, f.ring_v, static_cast<uint64_t>(S) * 8 * slots, 64, static_cast<uint32_t>(n_loaded), 64);
  if (rc != 0) return rc;
  const FrontArgs a = {f.x, f.ln_weight, f.ln_bias, static_cast<const uint16_t*>(f.w_qkv), f.cos, f.sin, f.cos_bstride, static_cast<uint16_t*>(f.ring_k),
                       static_cast<uint16_t*>(f.ring_v), static_cast<uint16_t*>(f.core), f.eps, scale * 1.4426950408889634f, f.stream_type, T, delta, slots, window,
                       (past - delta) % slots, past % slots, n_loaded};
  auto launch = [&](auto kern) {
    const int ok = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes), fmt = f.tc_fp16 ? 0 : 1;
    const uint32_t idesc = umma_idesc_f16(128, 16, fmt, fmt, 0, 0);
    return ok != 0 ? ok : launch_kernel(kern, dim3(static_cast<unsigned>(S) * 8), kThreads, kSmemBytes, st, 1, dependent, tk, tv, tw, a, idesc, status);
  };
  if (f.value_fp16) return f.tc_fp16 ? launch(stream_front_kernel<__half, __half>) : launch(stream_front_kernel<__half, __nv_bfloat16>);
  return f.tc_fp16 ? launch(stream_front_kernel<__nv_bfloat16, __half>) : launch(stream_front_kernel<__nv_bfloat16, __nv_bfloat16>);
}

}  // namespace fm
