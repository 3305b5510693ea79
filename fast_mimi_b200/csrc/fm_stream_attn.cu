// Attention of a few new frames per live stream over the stream's KV ring, and the ring's update, in one kernel
// (sm_100a).  T <= 8 new frames at positions past .. past + T - 1; q, k, v of the new frames come from the projection
// kernel as [S, T, 512], the ring [S, 8, slots, 64] holds position p in slot p % slots.
//
//   out[s, t, h, :] = softmax_p( scale * q . k_p ) v_p     over past + t - W < p <= past + t
//   ring slot (past + t) % slots <- new row t
//
// Covers the reference's cached attention of one or a few frames (MimiKVCache.update's concat-and-crop,
// src/fast_mimi/model.py:450-471, then SDPA with the band of src/fast_mimi/model.py:2194-2205).
//
// HBM-bound once there are more (stream, head) items than SMs, latency-bound below that.  An item is 2 x slots x 128
// bytes of ring; a persistent block streams items through shared memory (one TMA box each for K and V, 128-byte swizzle,
// up to three items in flight) and two groups of four warps take them in turn.  What limited the earlier forms was not
// the copy but the arithmetic around it: a dot product per lane, its conversions and shuffles cost 6400 warp instructions
// per item, half of the SM's issue slots at full bandwidth.  Here each warp multiplies its 64 slots with mma.sync
// (m16n8k16, FP32 accumulation): about 400 instructions per item, the same for one query as for eight, so a call of up to
// eight frames costs the ring's bytes once.  Keys and dimensions are the 16 rows of a product and the eight queries its
// columns: with the queries as rows half of every product was padding, and the chain of products (8 cycles each, 21 when
// one waits for the one before) was what a warp spent its time on (1024 streams, eight layers: 1082 us against 964).
// Probabilities keep the bits of FP32: they enter P V as sums of 16-bit parts.  (tcgen05 would need 128 rows and
// tensor-memory round trips for at most 8 queries.)
//
// Rows that are already in the ring do not depend on the projection, so in a chain of dependent launches the first items
// are requested before the wait for it.  A block has an item's ring rows in shared memory before it stores that item's
// new rows, and no other block touches its (stream, head): the ring is updated in place.
#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_stream_math.cuh"
#include "fm_warp_mma.cuh"

namespace fm {

namespace stream {
constexpr int kGroups = 2, kGroupWarps = 4;
constexpr int kThreads = (kGroups * kGroupWarps + 1) * 32;
constexpr int kMaxStages = 3;
constexpr int kMaxT = 8;
constexpr int kTileBytes = 256 * 128;                 // K or V of an item, padded to 256 slots
constexpr int kStageBytes = 2 * kTileBytes;
constexpr int kNewBytes = 2 * 16 * 128;               // new K and V rows of a group's item, padded to 16
constexpr int kMergeBytes = kGroupWarps * kMaxT * 64 * 4;
struct Ctl {
  // One "loaded" barrier per stage AND group: item n has barrier n % (2 stages), so that its phases are all waited for by
  // one group.  With one per stage and three stages the groups took a barrier's phases in turn, and a group that was done
  // with item n - 2 while item n - 3 was still on its way took the phase before that one for its own (the parity of a
  // phase cannot tell the one two before from it): it read, and gave back, a stage that was being filled.
  uint64_t full[kMaxStages * kGroups];
  uint64_t empty[kMaxStages];
  CtaCtl ctl;
  float m[kGroups][kGroupWarps][kMaxT];
  float l[kGroups][kGroupWarps][kMaxT];
};
constexpr int smem_bytes(int stages) { return 1024 + stages * kStageBytes + kGroups * (kNewBytes + kMergeBytes) + static_cast<int>(sizeof(Ctl)); }
static_assert(smem_bytes(kMaxStages) <= 232448, "exceeds the 227 KB a block may use");

}  // namespace stream

struct StreamArgs {
  const uint16_t *q, *k, *v;     // [S, T, 512]
  uint16_t *ring_k, *ring_v;     // [S, 8, slots, 64]
  uint16_t* out;                 // [S, T, 512]
  int n_items, T, past, delta, slots, window;
  int n_loaded;                  // ring rows per item that the tensor maps' boxes cover: min(past, slots)
  int stages;
  float scale_log2e;
};
// VT: type of the ring's values, v and the result
template <typename VT>
__global__ void __launch_bounds__(stream::kThreads, 1)
stream_attn_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ StreamArgs a, int* status) {
  using namespace stream;
  if (chain_stopped(status)) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_new = smem + a.stages * kStageBytes;
  float* smem_merge = reinterpret_cast<float*>(smem_new + kGroups * kNewBytes);
  Ctl* c = reinterpret_cast<Ctl*>(smem_new + kGroups * (kNewBytes + kMergeBytes));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(&c->empty[i], kGroupWarps);
    }
    for (int i = 0; i < kGroups * a.stages; ++i) mbar_init(&c->full[i], 1);
    c->ctl.abort = 0;
    fence_mbar_init();
  }
  // Slots past the loaded ones and rows past the new ones are never written: zeros, so that a probability of zero times
  // what lies there is zero.
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int i = threadIdx.x; i < a.stages * 2 * (256 - a.n_loaded) * 8; i += kThreads) {
    const int per = (256 - a.n_loaded) * 8, tile = i / per, piece = i % per;
    *reinterpret_cast<uint4*>(smem + tile * kTileBytes + a.n_loaded * 128 + piece * 16) = zero;
  }
  for (int i = threadIdx.x; i < kGroups * kNewBytes / 16; i += kThreads) *reinterpret_cast<uint4*>(smem_new + i * 16) = zero;
  fence_proxy_async_smem();
  __syncthreads();
  griddep_launch();
  CtaCtl* ctl = &c->ctl;

  if (warp == kGroups * kGroupWarps) {
    if (lane == 0) {
      if (a.n_loaded > 0) {
        tma_prefetch_desc(&tmap_k);
        tma_prefetch_desc(&tmap_v);
        int n = 0;
        for (int item = blockIdx.x; item < a.n_items; item += gridDim.x, ++n) {
          const int st = n % a.stages;
          mbar_wait(&c->empty[st], (static_cast<uint32_t>(n / a.stages) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
          uint64_t* full = &c->full[n % (kGroups * a.stages)];
          mbar_arrive_expect_tx(full, 2u * static_cast<uint32_t>(a.n_loaded) * 128u);
          tma_load_2d(smem + st * kStageBytes, &tmap_k, full, 0, item * a.slots);
          tma_load_2d(smem + st * kStageBytes + kTileBytes, &tmap_v, full, 0, item * a.slots);
        }
      }
      griddep_wait();
    }
  } else {
    griddep_wait();
    const int cg = warp / kGroupWarps, gw = warp % kGroupWarps, gt = threadIdx.x - cg * kGroupWarps * 32;
    const int g = lane >> 2, cpair = (lane & 3) * 2;     // mma fragments
    uint8_t* new_k = smem_new + cg * kNewBytes;
    uint8_t* new_v = new_k + kNewBytes / 2;
    float* merge = smem_merge + cg * (kMergeBytes / 4);
    const int first = a.slots > 0 ? (a.past - a.delta) % a.slots : 0;     // slot of the oldest visible row
    // An item's queries, straight into fragments (4 K-steps x {columns cpair.., cpair + 8..} of row g), and for the
    // group's last warp the new rows (16-byte pieces): asked for one item ahead, so that their latency passes behind the
    // item in hand.
    const int n_pieces = a.T * 8;
    uint32_t q_next[4][2];
    uint4 k_next[2], v_next[2];
    auto fetch = [&](long long item) {
      const size_t new0 = static_cast<size_t>(item >> 3) * a.T * 512 + static_cast<int>(item & 7) * 64;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          q_next[ks][e] = g < a.T ? __ldcg(reinterpret_cast<const uint32_t*>(a.q + new0 + static_cast<size_t>(g) * 512 + ks * 16 + e * 8 + cpair)) : 0u;
      }
      if (gw == kGroupWarps - 1) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int piece = lane + 32 * e;
          if (piece < n_pieces) {
            const size_t at = new0 + static_cast<size_t>(piece >> 3) * 512 + (piece & 7) * 8;
            k_next[e] = __ldcg(reinterpret_cast<const uint4*>(a.k + at));
            v_next[e] = __ldcg(reinterpret_cast<const uint4*>(a.v + at));
          }
        }
      }
    };
    auto take = [&](uint32_t (&qb)[4][2], uint4 (&nk)[2], uint4 (&nv)[2]) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) { qb[ks][0] = q_next[ks][0]; qb[ks][1] = q_next[ks][1]; }
#pragma unroll
      for (int e = 0; e < 2; ++e) { nk[e] = k_next[e]; nv[e] = v_next[e]; }
    };
    int n = cg;
    if (blockIdx.x + static_cast<long long>(cg) * gridDim.x < a.n_items) fetch(blockIdx.x + static_cast<long long>(cg) * gridDim.x);
    for (long long item = blockIdx.x + static_cast<long long>(cg) * gridDim.x; item < a.n_items;
         item += static_cast<long long>(kGroups) * gridDim.x, n += kGroups) {
      const int st = n % a.stages;
      const int s = static_cast<int>(item >> 3), h = static_cast<int>(item & 7);
      const size_t new0 = static_cast<size_t>(s) * a.T * 512 + h * 64;
      uint32_t qb[4][2];
      uint4 nk[2], nv[2];
      take(qb, nk, nv);
      if (item + static_cast<long long>(kGroups) * gridDim.x < a.n_items)
        fetch(item + static_cast<long long>(kGroups) * gridDim.x);
      if (a.n_loaded > 0)
        mbar_wait(&c->full[n % (kGroups * a.stages)], static_cast<uint32_t>(n / (kGroups * a.stages)) & 1u, ctl, status, kErrWaitTma);
      uint8_t* tile_k = smem + st * kStageBytes;
      uint8_t* tile_v = tile_k + kTileBytes;
      if (gw == kGroupWarps - 1) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int piece = lane + 32 * e, t = piece >> 3;
          if (piece < n_pieces) {
            *reinterpret_cast<uint4*>(new_k + sw128_offset(t, piece & 7)) = nk[e];
            *reinterpret_cast<uint4*>(new_v + sw128_offset(t, piece & 7)) = nv[e];
            if (t >= a.T - a.slots) {           // of two rows for one slot the newer stays
              const size_t at = (static_cast<size_t>(item) * a.slots + (a.past + t) % a.slots) * 64 + (piece & 7) * 8;
              *reinterpret_cast<uint4*>(a.ring_k + at) = nk[e];
              *reinterpret_cast<uint4*>(a.ring_v + at) = nv[e];
            }
          }
        }
        __syncwarp();
      }
      // Row number of slot j: its distance from the oldest visible row; rows >= delta are no longer visible to anyone.
      // What such a slot of V holds must not reach the sums through 0 * x.
      const int slot0 = gw * 64;
      {
        bool any = false;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = slot0 + lane + 32 * e;
          int r = j - first;
          if (r < 0) r += a.slots;
          if (j < a.n_loaded && r >= a.delta) {
            any = true;
#pragma unroll
            for (int p = 0; p < 8; ++p) *reinterpret_cast<uint4*>(tile_v + j * 128 + p * 16) = zero;
          }
        }
        if (__any_sync(0xffffffffu, any)) {
          fence_proxy_async_smem();                      // before the stage's next TMA load
          __syncwarp();
        }
      }

      // ---- scores, keys as rows: four tiles of 16 keys, and the new rows as a fifth for the group's last warp
      const int n_tiles = a.n_loaded > slot0 ? (a.n_loaded - slot0 + 15) >> 4 : 0;    // of four
      const bool has_new = gw == kGroupWarps - 1;
      auto in_use = [&](int mt) { return mt < 4 ? mt < n_tiles : has_new; };          // the same for the whole warp
      float sc[5][4];                                   // keys g (two queries) and g + 8 of each tile
#pragma unroll
      for (int mt = 0; mt < 5; ++mt) sc[mt][0] = sc[mt][1] = sc[mt][2] = sc[mt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
        for (int mt = 0; mt < 5; ++mt) {
          if (in_use(mt)) {
            uint32_t ka[4];                             // keys lane % 16, dimensions 16 ks + 8 (lane / 16) ..
            ldmatrix4(ka, smem_u32(mt < 4 ? tile_k : new_k) + sw128_offset((mt < 4 ? slot0 + mt * 16 : 0) + (lane & 15), 2 * ks + (lane >> 4)));
            mma_16x8x16<__nv_bfloat16>(sc[mt], ka, qb[ks][0], qb[ks][1]);
          }
        }
      }
      // visible rows of query t: delta + t - window < r <= delta + t
      float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
      for (int mt = 0; mt < 5; ++mt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int key = g + 8 * (e >> 1), t = cpair + (e & 1);
          int r;
          if (mt == 4) {
            r = a.delta + key;
          } else {
            const int j = slot0 + mt * 16 + key;
            r = j - first;
            if (r < 0) r += a.slots;
            if (j >= a.n_loaded || r >= a.delta) r = -(1 << 28);
          }
          const bool seen = in_use(mt) && r <= a.delta + t && r > a.delta + t - a.window;
          sc[mt][e] = seen ? sc[mt][e] * a.scale_log2e : -INFINITY;
          m[e & 1] = fmaxf(m[e & 1], sc[mt][e]);
        }
      }
      float m_use[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) m[e] = fmaxf(m[e], __shfl_xor_sync(0xffffffffu, m[e], x));
        m_use[e] = m[e] == -INFINITY ? 0.f : m[e] - Parts<VT>::kShift;
      }
#pragma unroll
      for (int mt = 0; mt < 5; ++mt) {
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

      // ---- O^T = V^T P^T, 16 keys per step, dimensions as rows.  A score fragment has keys along the lanes' groups and
      // queries inside them; as an operand it must be the other way round (movmatrix).
      float o[4][4];                                    // dimensions 16 d + g and + 8, two queries each
#pragma unroll
      for (int d = 0; d < 4; ++d) o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f;
#pragma unroll
      for (int mt = 0; mt < 5; ++mt) {
        if (in_use(mt)) {
          uint32_t p0[Parts<VT>::kParts], p1[Parts<VT>::kParts];
          split_pair<VT>(sc[mt][0], sc[mt][1], p0);
          split_pair<VT>(sc[mt][2], sc[mt][3], p1);
#pragma unroll
          for (int i = 0; i < Parts<VT>::kParts; ++i) {
            p0[i] = movmatrix_trans(p0[i]);
            p1[i] = movmatrix_trans(p1[i]);
          }
          const uint32_t base = smem_u32(mt < 4 ? tile_v : new_v);
          const int key = (mt < 4 ? slot0 + mt * 16 : 0) + (lane & 7) + ((lane >> 4) << 3);
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
      __syncwarp();
      if (lane == 0) mbar_arrive(&c->empty[st]);         // this warp's reads of the stage are done

      // ---- four-way merge
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = cpair + e;
        if (t < a.T) {
#pragma unroll
          for (int d = 0; d < 4; ++d) {
            merge[(gw * kMaxT + t) * 64 + d * 16 + g] = o[d][e];
            merge[(gw * kMaxT + t) * 64 + d * 16 + 8 + g] = o[d][2 + e];
          }
          if (g == 0) {
            c->m[cg][gw][t] = m[e];
            c->l[cg][gw][t] = l[e];
          }
        }
      }
      named_bar_sync(1 + cg, kGroupWarps * 32);
      for (int i = gt; i < a.T * 64; i += kGroupWarps * 32) {
        const int t = i >> 6, d = i & 63;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < kGroupWarps; ++w) mx = fmaxf(mx, c->m[cg][w][t]);
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < kGroupWarps; ++w) {
          const float f = ex2_approx(c->m[cg][w][t] - mx);            // 0 for a warp that saw no row
          num = fmaf(f, merge[(w * kMaxT + t) * 64 + d], num);
          den = fmaf(f, c->l[cg][w][t], den);
        }
        const size_t at = new0 + static_cast<size_t>(t) * 512 + d;
        const float y = num / den;
        a.out[at] = static_cast<uint16_t>(Pack16<VT>::pack(y, 0.f));
      }
      named_bar_sync(1 + cg, kGroupWarps * 32);          // the merge buffer and the new rows' tiles are free again
    }
  }
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);
}

int launch_stream_attn(const void* q, const void* k, const void* v, void* ring_k, void* ring_v, void* out, int S, int T,
                       int past, int slots, int window, float scale, int value_is_fp16, int* status,
                       cudaStream_t st, int dependent) {
  using namespace stream;
  if (S <= 0 || T <= 0) return (S == 0 || T == 0) ? 0 : -1;
  if (past < 0 || window <= 0 || slots < window || slots > 256 || T > kMaxT) return -1;
  if (static_cast<long long>(S) * 8 * slots > 0x7fffffffLL) return -1;      // a ring row is a coordinate of the tensor maps
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(ring_k) | reinterpret_cast<uintptr_t>(ring_v) | reinterpret_cast<uintptr_t>(out)) & 15u)
    return -3;
  const int delta = past < window - 1 ? past : window - 1;
  const int n_loaded = past < slots ? past : slots;
  CUtensorMap tk = {}, tv = {};
  if (n_loaded > 0) {
    int rc = encode_rows_16bit(&tk, ring_k, static_cast<uint64_t>(S) * 8 * slots, 64, static_cast<uint32_t>(n_loaded), 64);
    if (rc == 0) rc = encode_rows_16bit(&tv, ring_v, static_cast<uint64_t>(S) * 8 * slots, 64, static_cast<uint32_t>(n_loaded), 64);
    if (rc != 0) return rc;
  }
  const int n_items = S * 8, sms = sm_count();
  int stages = (n_items + sms - 1) / sms;               // one item per block: one stage, and room for other blocks
  if (stages > kMaxStages) stages = kMaxStages;
  const StreamArgs a = {static_cast<const uint16_t*>(q), static_cast<const uint16_t*>(k), static_cast<const uint16_t*>(v),
                  static_cast<uint16_t*>(ring_k), static_cast<uint16_t*>(ring_v), static_cast<uint16_t*>(out), n_items, T, past, delta, slots, window,
                  n_loaded, stages, scale * 1.4426950408889634f};
  const int bytes = smem_bytes(stages), blocks = n_items < sms ? n_items : sms;
  const auto kern = value_is_fp16 ? stream_attn_kernel<__half> : stream_attn_kernel<__nv_bfloat16>;
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), bytes);
  return rc != 0 ? rc : launch_kernel(kern, dim3(blocks), kThreads, bytes, st, 1, dependent, tk, tv, a, status);
}

}  // namespace fm
