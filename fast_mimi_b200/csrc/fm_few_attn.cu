// Banded causal attention for few query tiles (sm_100a): a clip or two, or chunks of more than eight frames on a handful
// of live streams, with the cached frames read from the ring where they lie.  Same contract as the tiled kernel
// (fm_prefill.cu): q, k, v [S, T, 512] rotated, query t of a stream sees the `window` newest frames up to its own, the
// min(past, window - 1) newest cached ones included (src/fast_mimi/model.py:1860-1868, :2194-2205, cache :450-471).
//
// Latency-bound.  The tcgen05 kernels give a block 128 queries and pass scores and probabilities through tensor memory
// with a hand-over between warps at every step: with 8 blocks on 148 SMs, 4.4 us for one tile of a 5 s clip, 13.5 us for
// a 50-frame chunk over a full ring.  Here a block has 64 or 32 queries and each of its eight warps carries 16 of them
// and a half or a quarter of every 64-key tile through the whole loop in registers (mma.sync m16n8k16, online softmax), so between
// the arrival of a tile and the next there is no barrier; the warps of the same queries meet once at the end.  (Four warps with whole tiles
// took 1.4 us per tile, a chain of latencies on one warp per scheduler.)  All tiles a chunk of up to 64 frames touches
// (five for a window of 250) are requested at once.
// Ring tiles do not depend on the projection and are requested before the wait for it; their slots are taken in slot
// order and the mask is derived from each slot's position, so nothing is copied into frame order first.  A chunk of up to 64
// frames also stores its new rows in the ring.
#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_warp_mma.cuh"

namespace fm {

namespace few {
constexpr int kTile = 64;                        // keys of a tile
constexpr int kTileBytes = kTile * 128;          // 8 KB
constexpr int kStages = 5;                       // K and V each
constexpr int kWarps = 8;                        // 16 queries each, of 64 or 32; so two or four share a tile's keys
constexpr int kThreads = (kWarps + 1) * 32;
struct Ctl {
  uint64_t q_full;
  uint64_t full[kStages];
  uint64_t empty[kStages];
  CtaCtl ctl;
};
constexpr int kMergeRow = 72;                     // 64 results, maximum and sum; fragments' pairs in different banks
constexpr int kSmemBytes = 1024 + kTileBytes + kStages * 2 * kTileBytes + 128;
static_assert(kWarps * 16 * kMergeRow * 4 <= kStages * 2 * kTileBytes, "the warps' results meet where the tiles lay");
static_assert(sizeof(Ctl) <= 128, "barrier block too large");
}  // namespace few

struct FewArgs {
  const uint16_t *k, *v;         // [S, T, 512], for the ring's update
  uint16_t *ring_k, *ring_v;     // [S, 8, slots, 64] or null
  uint16_t* out;                 // [S, T, 512]
  int T, past, delta, slots, window;
  int n_loaded;                  // slots of the ring that hold frames
  float scale_log2e;
};

// kQ: queries of a block, 64 or 32
template <typename VT, int kQ>
__global__ void __launch_bounds__(few::kThreads)
few_attn_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_rk,
                const __grid_constant__ CUtensorMap tmap_rv, const __grid_constant__ FewArgs a, int* status) {
  using namespace few;
  constexpr int kQWarps = kQ / 16, kGroups = kWarps / kQWarps, kKeys = kTile / kGroups;      // kKeys: of a tile, a warp
  if (chain_stopped(status)) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_q = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_kv = smem_q + kTileBytes;
  float* merge = reinterpret_cast<float*>(smem_kv);
  Ctl* c = reinterpret_cast<Ctl*>(smem_kv + kStages * 2 * kTileBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = static_cast<int>(blockIdx.x) * kQ, h = static_cast<int>(blockIdx.y), s = static_cast<int>(blockIdx.z);
  if (threadIdx.x == 0) {
    mbar_init(&c->q_full, 1);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&c->full[i], 1);
      mbar_init(&c->empty[i], kWarps);
    }
    c->ctl.abort = 0;
    fence_mbar_init();
  }
  __syncthreads();
  griddep_launch();
  CtaCtl* ctl = &c->ctl;

  // Rows on the key axis: cached rows 0 .. delta - 1, then the new rows.  Query t sees rows (delta + t - window, delta + t].
  // This block's band:
  const int q_last = (q0 + kQ < a.T ? q0 + kQ : a.T) - 1;
  const int band_lo = a.delta + q0 - a.window + 1, band_hi = a.delta + q_last;
  const int first = a.delta > 0 ? (a.past - a.delta) % a.slots : 0;        // slot of row 0
  // Ring tile i: slots 64 i ...  Their rows run in at most two pieces; the tile is left out if no row of it is in the band.
  auto ring_row = [&](int slot) {
    int r = slot - first;
    return r < 0 ? r + a.slots : r;
  };
  auto ring_tile_visible = [&](int i) {
    const int lo = i * kTile, hi = (lo + kTile < a.n_loaded ? lo + kTile : a.n_loaded) - 1;
    if (lo > hi) return false;
    // the newest cached row of the tile
    const int newest = (first > lo && first <= hi) ? ring_row(first - 1) : ring_row(hi);
    const int oldest = (first >= lo && first <= hi) ? 0 : ring_row(lo);
    return newest >= band_lo && oldest < a.delta;
  };
  const int n_ring = a.delta > 0 ? (a.n_loaded + kTile - 1) / kTile : 0;
  const int new_lo = band_lo - a.delta > 0 ? (band_lo - a.delta) / kTile : 0, new_hi = (band_hi - a.delta) / kTile;

  if (warp == kWarps) {
    if (lane == 0) {
      int n = 0;
      auto open_stage = [&]() {
        const int st = n % kStages;
        mbar_wait(&c->empty[st], (static_cast<uint32_t>(n / kStages) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
        mbar_arrive_expect_tx(&c->full[st], 2 * kTileBytes);
        ++n;
        return st;
      };
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      for (int i = 0; i < n_ring; ++i) {
        if (!ring_tile_visible(i)) continue;
        const int st = open_stage();
        tma_load_3d(smem_kv + 2 * st * kTileBytes, &tmap_rk, &c->full[st], 0, i * kTile, s * 8 + h);
        tma_load_3d(smem_kv + (2 * st + 1) * kTileBytes, &tmap_rv, &c->full[st], 0, i * kTile, s * 8 + h);
        if (n == kStages) break;           // the rest after the queries are on their way
      }
      const int early = n;
      griddep_wait();
      mbar_arrive_expect_tx(&c->q_full, kQ * 128);
      tma_load_3d(smem_q, &tmap_q, &c->q_full, h * 64, q0, s);
      int seen = 0;
      for (int i = 0; i < n_ring; ++i) {
        if (!ring_tile_visible(i) || seen++ < early) continue;
        const int st = open_stage();
        tma_load_3d(smem_kv + 2 * st * kTileBytes, &tmap_rk, &c->full[st], 0, i * kTile, s * 8 + h);
        tma_load_3d(smem_kv + (2 * st + 1) * kTileBytes, &tmap_rv, &c->full[st], 0, i * kTile, s * 8 + h);
      }
      for (int j = new_lo; j <= new_hi; ++j) {
        const int st = open_stage();
        tma_load_3d(smem_kv + 2 * st * kTileBytes, &tmap_k, &c->full[st], h * 64, j * kTile, s);
        tma_load_3d(smem_kv + (2 * st + 1) * kTileBytes, &tmap_v, &c->full[st], h * 64, j * kTile, s);
      }
    }
    __syncwarp();
  } else {
    griddep_wait();
    const int g = lane >> 2, cpair = (lane & 3) * 2;      // fragments: rows g and g + 8 of the warp's 16, columns cpair, + 1
    const int qw = warp % kQWarps, key0 = warp / kQWarps * kKeys;     // 16 queries, kKeys of every tile
    mbar_wait(&c->q_full, 0, ctl, status, kErrWaitTma);
    uint32_t qa[4][4];
    {
      // x4: rows lane % 16, 16-byte piece 2 ks + lane / 16
      const uint32_t base = smem_u32(smem_q);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) ldmatrix4(qa[ks], base + sw128_offset(qw * 16 + (lane & 15), 2 * ks + (lane >> 4)));
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    float o[8][4];
#pragma unroll
    for (int d = 0; d < 8; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
    const int row_hi[2] = {a.delta + q0 + qw * 16 + g, a.delta + q0 + qw * 16 + g + 8};   // newest row a query sees
    const int warp_lo = a.delta + q0 + qw * 16 - a.window + 1, warp_hi = a.delta + q0 + qw * 16 + 15;
    int n = 0;
    // One 64-key tile; row_of(column) gives a key's row, or a number below every band for a slot nobody sees.
    auto tile = [&](auto row_of, bool all_visible, bool any_visible, bool from_ring) {
      const int st = n % kStages;
      mbar_wait(&c->full[st], static_cast<uint32_t>(n / kStages) & 1u, ctl, status, kErrWaitTma);
      ++n;
      if (any_visible) {
        const uint32_t kb = smem_u32(smem_kv + 2 * st * kTileBytes), vb = kb + kTileBytes;
        if (from_ring) {
          // What a slot outside the window holds must not reach the sums as 0 * x: one in a full ring of `window` slots,
          // any number, and frames long past in a ring not yet full, where it has more.  Every warp clears those of its keys.
          const bool gone = lane < kKeys && row_of(key0 + lane % kKeys) < 0;
          if (gone) {
#pragma unroll
            for (int p = 0; p < 8; ++p)
              *reinterpret_cast<uint4*>(smem_kv + (2 * st + 1) * kTileBytes + (key0 + lane) * 128 + p * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          if (__any_sync(0xffffffffu, gone)) {
            fence_proxy_async_smem();                    // before the stage's next TMA load
            __syncwarp();
          }
        }
        float sc[kKeys / 8][4];
#pragma unroll
        for (int nt = 0; nt < kKeys / 8; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
        for (int half = 0; half < 2; ++half) {           // dimensions 0 .. 31, 32 .. 63; independent products in a row
          uint32_t b[kKeys / 8][4];
#pragma unroll
          for (int nt = 0; nt < kKeys / 8; ++nt) ldmatrix4(b[nt], kb + sw128_offset(key0 + nt * 8 + (lane & 7), 4 * half + (lane >> 3)));
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
            for (int nt = 0; nt < kKeys / 8; ++nt) mma_16x8x16<__nv_bfloat16>(sc[nt], qa[2 * half + ks], b[nt][2 * ks], b[nt][2 * ks + 1]);
          }
        }
        float m_new[2] = {m[0], m[1]};
#pragma unroll
        for (int nt = 0; nt < kKeys / 8; ++nt) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float x = sc[nt][e] * a.scale_log2e;
            if (!all_visible) {
              const int r = row_of(key0 + nt * 8 + cpair + (e & 1));
              if (r > row_hi[e >> 1] || r <= row_hi[e >> 1] - a.window) x = -INFINITY;
            }
            sc[nt][e] = x;
            m_new[e >> 1] = fmaxf(m_new[e >> 1], x);
          }
        }
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          m_new[r] = fmaxf(m_new[r], __shfl_xor_sync(0xffffffffu, m_new[r], 1));
          m_new[r] = fmaxf(m_new[r], __shfl_xor_sync(0xffffffffu, m_new[r], 2));
          const float use = m_new[r] == -INFINITY ? 0.f : m_new[r];
          alpha[r] = ex2_approx(m[r] - use);            // 0 while nothing has been seen yet
          m[r] = m_new[r];
          m_new[r] = use;
          l[r] *= alpha[r];
        }
#pragma unroll
        for (int d = 0; d < 8; ++d) {
          o[d][0] *= alpha[0]; o[d][1] *= alpha[0]; o[d][2] *= alpha[1]; o[d][3] *= alpha[1];
        }
#pragma unroll
        for (int ks = 0; ks < kKeys / 16; ++ks) {
          float p[2][4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              p[u][e] = ex2_approx(sc[2 * ks + u][e] - m_new[e >> 1]);
              l[e >> 1] += p[u][e];
            }
          }
          const uint32_t pa[4] = {Pack16<VT>::pack(p[0][0], p[0][1]), Pack16<VT>::pack(p[0][2], p[0][3]),
                                  Pack16<VT>::pack(p[1][0], p[1][1]), Pack16<VT>::pack(p[1][2], p[1][3])};
#pragma unroll
          for (int dp = 0; dp < 4; ++dp) {
            uint32_t b[4];
            ldmatrix4_trans(b, vb + sw128_offset(key0 + ks * 16 + (lane & 15), dp * 2 + (lane >> 4)));
            mma_16x8x16<VT>(o[2 * dp], pa, b[0], b[1]);
            mma_16x8x16<VT>(o[2 * dp + 1], pa, b[2], b[3]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&c->empty[st]);
    };
    for (int i = 0; i < n_ring; ++i) {
      if (!ring_tile_visible(i)) continue;
      tile([&](int col) {
        const int slot = i * kTile + col;
        const int r = ring_row(slot);
        return slot >= a.n_loaded || r >= a.delta ? -(1 << 28) : r;
      }, false, true, true);
    }
    for (int j = new_lo; j <= new_hi; ++j) {
      const int r0 = a.delta + j * kTile;
      tile([&](int col) { return r0 + col; }, r0 + kTile - 1 <= a.delta + q0 + qw * 16 && r0 > warp_hi - a.window,
           r0 + key0 <= warp_hi && r0 + key0 + kKeys - 1 >= warp_lo, false);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    // ---- the warps with the same queries meet where the tiles lay; each normalises and rounds its share of their dimensions
    named_bar_sync(1, kWarps * 32);
    {
      float* mine = merge + warp * 16 * kMergeRow;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int d = 0; d < 8; ++d)
          *reinterpret_cast<float2*>(mine + (g + 8 * r) * kMergeRow + d * 8 + cpair) = make_float2(o[d][2 * r], o[d][2 * r + 1]);
        if ((lane & 3) == 0) *reinterpret_cast<float2*>(mine + (g + 8 * r) * kMergeRow + 64) = make_float2(m[r], l[r]);
      }
    }
    named_bar_sync(1, kWarps * 32);
    // eight results of a row a thread
#pragma unroll
    for (int item = static_cast<int>(threadIdx.x); item < kQ * 8; item += kWarps * 32) {
      const int row = item >> 3, piece = item & 7, t = q0 + row;
      const float* first = merge + row * kMergeRow;
      float2 ml[kGroups];
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        ml[i] = *reinterpret_cast<const float2*>(first + i * kQ * kMergeRow + 64);
        mx = fmaxf(mx, ml[i].x);
      }
      const float use = mx == -INFINITY ? 0.f : mx;
      float x[8] = {}, den = 0.f;
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        const float f = ex2_approx(ml[i].x - use);     // 0 for a warp that saw nothing
        den += f * ml[i].y;
        const float4* v = reinterpret_cast<const float4*>(first + i * kQ * kMergeRow + piece * 8);
        const float4 lo = v[0], hi = v[1];
        x[0] += f * lo.x; x[1] += f * lo.y; x[2] += f * lo.z; x[3] += f * lo.w;
        x[4] += f * hi.x; x[5] += f * hi.y; x[6] += f * hi.z; x[7] += f * hi.w;
      }
      const float inv = 1.f / den;
      if (t < a.T)
        *reinterpret_cast<uint4*>(a.out + (static_cast<size_t>(s) * a.T + t) * 512 + h * 64 + piece * 8) =
            make_uint4(Pack16<VT>::pack(x[0] * inv, x[1] * inv), Pack16<VT>::pack(x[2] * inv, x[3] * inv), Pack16<VT>::pack(x[4] * inv, x[5] * inv),
                       Pack16<VT>::pack(x[6] * inv, x[7] * inv));
    }
  }
  __syncthreads();
  griddep_wait();
  if (a.ring_k != nullptr && a.T <= kTile) {
    // every ring tile this (stream, head) reads has landed, in its other block too: the new rows take their slots
    if (gridDim.x > 1) cluster_sync_all();
    for (int i = static_cast<int>(blockIdx.x) * kThreads + threadIdx.x; i < a.T * 8; i += gridDim.x * kThreads) {
      const int t = i >> 3;
      if (t < a.T - a.slots) continue;                   // of two rows for one slot the newer stays
      const size_t src = (static_cast<size_t>(s) * a.T + t) * 512 + h * 64 + (i & 7) * 8;
      const size_t dst = ((static_cast<size_t>(s) * 8 + h) * a.slots + (a.past + t) % a.slots) * 64 + (i & 7) * 8;
      *reinterpret_cast<uint4*>(a.ring_k + dst) = __ldcg(reinterpret_cast<const uint4*>(a.k + src));
      *reinterpret_cast<uint4*>(a.ring_v + dst) = __ldcg(reinterpret_cast<const uint4*>(a.v + src));
    }
  }
  if (ctl->abort) __nanosleep(20000);
}

bool few_attn_tiles(int S, int T) { return static_cast<long long>(S) * 8 * ((T + few::kTile - 1) / few::kTile) <= 2ll * sm_count(); }
bool few_attn_updates_ring(int T) { return T <= few::kTile; }

int launch_few_attn(const void* q, const void* k, const void* v, void* ring_k, void* ring_v, void* out, int S, int T, int past,
                    int slots, int window, float scale, int value_is_fp16, int* status, cudaStream_t st, int dependent) {
  using namespace few;
  if (S <= 0 || T <= 0) return (S == 0 || T == 0) ? 0 : -1;
  if (window <= 0 || S > 65535 || past < 0) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(ring_k) | reinterpret_cast<uintptr_t>(ring_v) | reinterpret_cast<uintptr_t>(out)) & 15u)
    return -3;
  const bool cached = ring_k != nullptr;
  const int delta = cached ? (past < window - 1 ? past : window - 1) : 0;
  if (cached && slots < window) return -1;
  const int n_loaded = cached ? (past < slots ? past : slots) : 0;
  // 32 queries a block as far as every block has an SM then: mma.sync takes 16 cycles an instruction and scheduler, so that a tile costs half,
  // and the warps that share it are twice as many (eight layers: clip of 125 frames 157 -> 150 us, two of 100 201 -> 188, five streams of 50 frames
  // 230 -> 216; 9 of 64, 144 blocks, 286 -> 297).  Two blocks that share a ring are a cluster, which pays up to about half of the SMs (80 blocks 230 -> 217, 96 243 ->
  // 246, 128 243 -> 252).  One clip of up to 64 frames keeps to eight blocks: sixteen leave the clusters behind them fewer GPCs with SMs enough
  // (41 frames 98 -> 106, 50 frames 108 -> 109, 64 frames 113 -> 111).
  const int sms = sm_count(), narrow = S * 8 * ((T + 31) / 32), shares_ring = cached && T > 32 && T <= kTile;
  const bool one_clip = !cached && S == 1 && T > 32 && T <= kTile;
  const int queries = S <= sms && !one_clip && narrow <= (shares_ring ? sms * 9 / 16 : sms) ? 32 : 64;
  auto frames = [&](CUtensorMap* map, const void* base, int rows) {
    const cuuint64_t dims[3] = {512, static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(S)};
    const cuuint64_t strides[2] = {1024, static_cast<cuuint64_t>(T) * 1024};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(rows), 1}, estr[3] = {1, 1, 1};
    return encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  };
  auto ring = [&](CUtensorMap* map, const void* base) {      // rows past the filled slots read as zero
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(n_loaded), static_cast<cuuint64_t>(S) * 8};
    const cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(slots) * 128};
    const cuuint32_t box[3] = {64, kTile, 1}, estr[3] = {1, 1, 1};
    return encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  };
  CUtensorMap tq, tk, tv, trk = {}, trv = {};
  int rc = frames(&tq, q, queries);
  if (rc == 0) rc = frames(&tk, k, kTile);
  if (rc == 0) rc = frames(&tv, v, kTile);
  if (rc == 0 && delta > 0) rc = ring(&trk, ring_k);
  if (rc == 0 && delta > 0) rc = ring(&trv, ring_v);
  if (rc != 0) return rc;
  const FewArgs a = {static_cast<const uint16_t*>(k), static_cast<const uint16_t*>(v), static_cast<uint16_t*>(ring_k),
                     static_cast<uint16_t*>(ring_v), static_cast<uint16_t*>(out), T, past, delta, slots, window, n_loaded,
                     scale * 1.4426950408889634f};
  auto kern = queries == 32 ? (value_is_fp16 ? few_attn_kernel<__half, 32> : few_attn_kernel<__nv_bfloat16, 32>)
                            : (value_is_fp16 ? few_attn_kernel<__half, 64> : few_attn_kernel<__nv_bfloat16, 64>);
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes);
  if (rc != 0) return rc;
  const int tiles = (T + queries - 1) / queries, cluster = cached && T <= kTile && tiles > 1 ? tiles : 1;
  return launch_kernel(kern, dim3(tiles, 8, S), kThreads, kSmemBytes, st, cluster, dependent, tq, tk, tv, trk, trv, a, status);
}

}  // namespace fm
