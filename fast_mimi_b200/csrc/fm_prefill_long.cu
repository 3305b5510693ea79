// Banded causal attention for long clips (T > 256 frames) with a window of 130..257 frames (Mimi: 250), sm_100a.
// Same contract as the general prefill kernel (fm_prefill.cu): rotated q, k (BF16) and v (16-bit) in
// [B, T, 512], output [B, T, 512]; replaces the masked SDPA call of the reference
// (src/fast_mimi/model.py:1860-1868 with the band of src/fast_mimi/model.py:1672-1676) for long sequences.
//
// With such a window the 128 queries of tile t see keys of exactly three 128-key tiles: t-2 (far), t-1 (mid)
// and t (diagonal).  A persistent CTA walks RUNS of consecutive query tiles of one (clip, head), so the K and
// V tiles it needs are already in shared memory from the previous two steps: a ring of four K tiles and four
// V tiles (tile u in slot u % 4); per step it loads only Q_t, K_t and V_t (48 KB for 128 frames), each byte
// once.  A run's first step also loads its two halo tiles.
//
// The step's three 128 x 128 score tiles are three JOBS: far, mid and diagonal, each with 128 columns of tensor memory and a softmax
// team of four warps of its own; S = Q K^T is turned in place into 16-bit P, which the tensor core reads from tensor memory for
// O = P V.  All three jobs belong to the same 128 query rows: the teams exchange row maxima through shared memory, use one common
// maximum, and the tensor core adds the three P V products into one of two accumulators beside the jobs' columns.  So a job's next
// scores follow as soon as its own P has been read, and a fourth team normalises and stores the rows behind the others' backs.  (With
// O in the diagonal job's columns and four columns' sets for three jobs in turn, a step held its columns until its last row was out:
// 16 FP16 clips of 2500 frames, 18 steps a block, 107 us, now 98, of which 3 by the tests in fm_attn_tile.cuh.)  The window gives warp w of the
// far job 4-w visible 32-key groups and warp w of the diagonal job w+1, so the four SM sub-partitions carry
// the same load.  Tiles before the clip's first frame are not loaded; their jobs run empty.
// Warps 0-11: softmax teams.  Warps 12-15: results.  Warp 16: Q/K loads + score products.  Warp 17: P V products.  Warp 18: V loads.
//
// FP32 q, k, v (a model's own, any strides) of calls with some steps a block are converted on the way: pieces of 16 rows arrive by TMA in a staging
// buffer, three for each of four warps (18 to 21), which round them (q, k to BF16, v to its type) into the tiles' places.  The
// kernel is bound by its chain of steps, not by memory, so the 12 bytes a value triple costs instead of 6 pass behind it; a
// converting pass in front (18 bytes a triple at the copy rate) took 51 of 141 us for 16 clips of 2500 frames, 25 clips of 1500
// frames 132; now 91 and 87 (two warps, which kept the others waiting once those had become faster: 104 and 98).  What counts is the
// little they do besides (a proxy fence, an index division and a walk of its own for every piece: 141 us instead of 107 with two).
#include "fm_attn_tile.cuh"
#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_shares.h"

namespace fm {

namespace longclip {
using attn_tile::kD;
using attn_tile::kTile;
constexpr int kTileBytes = kTile * kD * 2;          // 16 KB
constexpr int kSlabBytes = 32 * 128;                // 32 rows x 64 x 16 bit
constexpr int kJobs = 3;
constexpr int kRing = 4;                            // K tiles and V tiles kept: t-2, t-1, t and the next step's
constexpr int kSoftmaxWarps = 4 * (kJobs + 1);      // and those that store
constexpr int kIssueWarps = 3;
constexpr int kThreads = (kSoftmaxWarps + kIssueWarps) * 32;
constexpr int kTmemCols = 512;
constexpr uint32_t kOCol = 128 * kJobs;             // three jobs' scores, P over them; then two steps' O

// FP32 inputs: staged pieces of tiles, two of a tile for each converting warp
constexpr int kConvertWarps = 4, kStaged = 3;
constexpr int kPieceRows = kTile / (2 * kConvertWarps), kPieceBytes = kPieceRows * kD * 4;
constexpr int threads(bool f32_in) { return kThreads + (f32_in ? (kConvertWarps - 1) * 32 : 0); }

struct Shared {
  uint64_t staged[kConvertWarps][kStaged];   // a piece has landed
  uint64_t qk_full[2];     // Q and the new K tile(s) of the step in this Q buffer have landed
  uint64_t v_full[2];      // the new V tile(s) of the step have landed
  uint64_t qk_done[2];     // the step's score products have completed: its Q buffer and its far K tile are dead
  uint64_t pv_done[2];     // the step's P V products have completed: its far V tile is dead, its O is there
  uint64_t o_free[2];      // O has been read
  uint64_t s_full[kJobs];  // by job, a phase a step
  uint64_t p_full[kJobs];
  uint64_t p_done[kJobs];  // the P V product that reads P has completed
  uint64_t xm_full[4];     // the three partial row maxima of a step are published (12 warps)
  uint64_t xl_full[4];     // the row sums of the three jobs are published (12 warps)
  uint32_t tmem_base;
  CtaCtl ctl;
  float xm[4][kTile][3];   // by step % 4
  float xl[4][kTile][3];
};
__host__ __device__ constexpr int stage_bytes(bool f32_in) { return f32_in ? kConvertWarps * kStaged * kPieceBytes : 4 * kSlabBytes; }
constexpr int smem_bytes(bool f32_in) {
  return 1024 + 2 * kRing * kTileBytes + 2 * kTileBytes + stage_bytes(f32_in) + static_cast<int>((sizeof(Shared) + 127) & ~size_t(127));
}
static_assert(smem_bytes(true) <= 232448, "exceeds the 227 KB a CTA may use");

// The steps a CTA takes: an equal share of all (clip, head, query tile) triples in that order (fm_shares.h), i.e. at most a rest of
// one sequence, whole ones, and the beginning of another; each of those is a run.  (Whole sequences dealt out in turn: 128 sequences
// of 20 tiles took 20 steps on 128 of 148 SMs, now 18 at most, 200 sequences of 12 tiles 24 steps, now 17; 16 FP16 clips of 2500 frames 116.6 ->
// 107.2 us with the chain of steps of then, which takes 98 now.)  A run re-reads the two K / V tiles in front of it and its first step waits for
// all of them, so shares keep to sequences where that takes no block more steps: rounded to occupy every SM, they began anywhere (9 FP16
// clips of 513 frames 20.4 us, with segments of each sequence 18.6, both of then).  Every role of the kernel walks the same steps with the
// same counter n, which the barrier phases are derived from.
struct Walk {
  int n_tiles, seq, t, t0, n, steps;
  __device__ __forceinline__ explicit Walk(const Shares& shares) : n_tiles(shares.tiles), n(0) {
    shares.share(static_cast<int>(blockIdx.x), &seq, &t, &steps);
    t0 = t;
  }
  __device__ __forceinline__ bool valid() const { return n < steps; }
  __device__ __forceinline__ bool first() const { return t == t0; }
  __device__ __forceinline__ int clip() const { return seq >> 3; }
  __device__ __forceinline__ int head() const { return seq & 7; }
  __device__ __forceinline__ int first_tile_loaded() const { return t0 - 2 > 0 ? t0 - 2 : 0; }   // run's oldest halo tile
  __device__ __forceinline__ void next() {
    ++n;
    if (++t == n_tiles) {
      t = t0 = 0;
      ++seq;
    }
  }
};
}  // namespace longclip

// OT: type of the result.  FP32 rows (256 bytes per lane) go straight from registers to memory as whole 32-byte sectors;
// 16-bit rows through the slabs and a tiled store.
// kF32In: q, k, v are FP32 (the result too).
template <typename VT, typename OT, bool kF32In>
__global__ void __launch_bounds__(longclip::threads(kF32In), 1)
band_attn_long_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_out,
                      float* __restrict__ out32, const __grid_constant__ Shares shares, int T, int window, float scale_log2e,
                      int* status) {
  using namespace longclip;
  using namespace attn_tile;
  if (chain_stopped(status)) return;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_k = smem;                              // kRing tiles
  uint8_t* smem_v = smem_k + kRing * kTileBytes;       // kRing tiles
  uint8_t* smem_q = smem_v + kRing * kTileBytes;       // two tiles
  uint8_t* smem_stage = smem_q + 2 * kTileBytes;       // four slabs, or staged FP32 pieces
  Shared* sh = reinterpret_cast<Shared*>(smem_stage + stage_bytes(kF32In));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->qk_full[i], kF32In ? kConvertWarps : 1);
      mbar_init(&sh->v_full[i], kF32In ? kConvertWarps : 1);
      mbar_init(&sh->qk_done[i], 1);
      mbar_init(&sh->pv_done[i], 1);
      mbar_init(&sh->o_free[i], 4);
    }
    for (int i = 0; i < kJobs; ++i) {
      mbar_init(&sh->s_full[i], 1);
      mbar_init(&sh->p_full[i], 4);
      mbar_init(&sh->p_done[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&sh->xm_full[i], 12);
      mbar_init(&sh->xl_full[i], 12);
    }
    for (int i = 0; kF32In && i < kConvertWarps * kStaged; ++i) mbar_init(&sh->staged[i / kStaged][i % kStaged], 1);
    sh->ctl.abort = 0;
    fence_mbar_init();
  }
  if (warp == kSoftmaxWarps) {
    tmem_alloc(&sh->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  griddep_launch();
  griddep_wait();                       // q, k, v may come from the kernel in front
  const uint32_t tmem_base = sh->tmem_base;
  CtaCtl* ctl = &sh->ctl;

  auto step_phase = [](int n) { return static_cast<uint32_t>(n >> 1) & 1u; };

  if (warp >= kSoftmaxWarps) {
    // All 32 lanes of an issuing warp walk its loop and one elected lane issues copies, MMAs and commits:
    // warp-uniform control flow keeps the descriptors in uniform registers and the sequences issue faster than
    // from a single lane under a lane test.
    const int role = warp - kSoftmaxWarps;
    const bool one = elect_one();
    constexpr uint32_t idesc_qk = umma_idesc_f16(kTile, kTile, 1, 1, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_f16(kTile, kD, Pack16<VT>::kFmt, Pack16<VT>::kFmt, 0, 1);
    auto job_addr = [&](int kind) { return tmem_base + static_cast<uint32_t>(kind * kTile); };
    auto out_addr = [&](int n) { return tmem_base + kOCol + static_cast<uint32_t>((n & 1) * kD); };
    if (role == 0) {
      // ---------------------------------------------------------- Q / K loads + score products
      if (!kF32In && one) {
        tma_prefetch_desc(&tmap_q);
        tma_prefetch_desc(&tmap_k);
      }
      auto load_qk = [&](const Walk& w) {
        if (kF32In || !one) return;
        const int b = w.n & 1;
        const int u_lo = w.first() ? w.first_tile_loaded() : w.t;     // K tiles u_lo .. t arrive with this step
        mbar_arrive_expect_tx(&sh->qk_full[b], static_cast<uint32_t>((w.t - u_lo + 2) * kTileBytes));
        tma_load_3d(smem_q + b * kTileBytes, &tmap_q, &sh->qk_full[b], w.head() * kD, w.t * kTile, w.clip());
        for (int u = u_lo; u <= w.t; ++u)
          tma_load_3d(smem_k + (u & 3) * kTileBytes, &tmap_k, &sh->qk_full[b], w.head() * kD, u * kTile, w.clip());
      };
      Walk cur(shares), nxt = cur;
      if (cur.valid()) {
        load_qk(cur);
        nxt.next();
      }
      for (; cur.valid(); cur.next(), nxt.next()) {
        const int n = cur.n;
        if (nxt.valid() && !nxt.first()) {
          // Step n+1 of the same run reuses the Q buffer of step n-1 and the ring slot of that step's far
          // tile; both are dead once step n-1's scores exist.
          if (n >= 1) mbar_wait(&sh->qk_done[(n + 1) & 1], step_phase(n - 1), ctl, status, kErrWaitMma);
          load_qk(nxt);
        }
        mbar_wait(&sh->qk_full[n & 1], step_phase(n), ctl, status, kErrWaitTma);
        const uint64_t qd = umma_desc_sw128(smem_u32(smem_q + (n & 1) * kTileBytes));
        for (int kind = 0; kind < 3; ++kind) {
          // the job's columns: its P of the step before has been read
          if (n >= 1) mbar_wait(&sh->p_done[kind], static_cast<uint32_t>(n - 1) & 1u, ctl, status, kErrWaitMma);
          tc_fence_after_sync();
          const int u = cur.t - 2 + kind;              // key tile of this job
          if (u >= 0) {
            const uint64_t kd = umma_desc_sw128(smem_u32(smem_k + (u & 3) * kTileBytes));
#pragma unroll
            for (int ks = 0; ks < kD / 16; ++ks)
              if (one) tc_mma_ss(job_addr(kind), qd + 2u * ks, kd + 2u * ks, idesc_qk, ks != 0);
          }
          if (one) {
            tc_commit(&sh->s_full[kind]);
            if (kind == 2) tc_commit(&sh->qk_done[n & 1]);
          }
        }
        if (nxt.valid() && nxt.first()) {
          // A new run: its tiles go into ring slots that this step's tiles may still occupy.
          mbar_wait(&sh->qk_done[n & 1], step_phase(n), ctl, status, kErrWaitMma);
          load_qk(nxt);
        }
      }
    } else if (role == 1) {
      // ---------------------------------------------------------- P V products
      for (Walk w(shares); w.valid(); w.next()) {
        const int n = w.n;
        mbar_wait(&sh->v_full[n & 1], step_phase(n), ctl, status, kErrWaitTma);
        mbar_wait(&sh->o_free[n & 1], step_phase(n) ^ 1u, ctl, status, kErrWaitConsumer);
        bool accumulate = false;
        for (int kind = 0; kind < 3; ++kind) {
          mbar_wait(&sh->p_full[kind], static_cast<uint32_t>(n) & 1u, ctl, status, kErrWaitConsumer);
          tc_fence_after_sync();
          const int u = w.t - 2 + kind;
          if (u >= 0) {
            // O (+)= P V: A = P from tensor memory (8 columns per 16 keys), B = V (MN-major, 2 KB per 16 keys)
            const uint64_t v = umma_desc_sw128(smem_u32(smem_v + (u & 3) * kTileBytes));
#pragma unroll
            for (int ks = 0; ks < kTile / 16; ++ks)
              if (one)
                tc_mma_ts(out_addr(n), job_addr(kind) + 8u * ks, v + static_cast<uint64_t>(ks) * 128u, idesc_pv, (accumulate || ks != 0) ? 1u : 0u);
            accumulate = true;
          }
          if (one) tc_commit(&sh->p_done[kind]);
        }
        if (one) tc_commit(&sh->pv_done[n & 1]);
      }
    } else if (kF32In) {
      // ---------------------------------------------------------- FP32 tiles into their places (four warps)
      // A step's tiles in the order of their use: its new K tiles and Q, then its new V tiles; this warp has pieces 2c and
      // 2c + 1 of each.  Copies run kStaged pieces ahead of the conversion.
      const int c = role - 2;
      uint8_t* staging = smem_stage + c * kStaged * kPieceBytes;
      // Copies: their own walk, with what a run's tiles have in common worked out once.
      Walk to_ask(shares);
      int ask_nk = 0, ask_tile = 0, ask_half = 0, ask_head = 0, ask_clip = 0, asked = 0;
      auto open_step = [&]() {
        if (to_ask.first()) {
          ask_head = to_ask.head();
          ask_clip = to_ask.clip();
        }
        ask_nk = to_ask.first() ? to_ask.t - to_ask.first_tile_loaded() + 1 : 1;
      };
      open_step();
      auto ask = [&]() {
        if (!to_ask.valid()) return;
        const CUtensorMap* map = ask_tile < ask_nk ? &tmap_k : (ask_tile == ask_nk ? &tmap_q : &tmap_v);
        const int u = to_ask.t - (ask_tile < ask_nk ? ask_nk - 1 - ask_tile : (ask_tile == ask_nk ? 0 : 2 * ask_nk - ask_tile));
        if (one) {
          uint64_t* bar = &sh->staged[c][asked];
          mbar_arrive_expect_tx(bar, kPieceBytes);
          tma_load_4d(staging + asked * kPieceBytes, map, bar, 0, u * kTile + (2 * c + ask_half) * kPieceRows, ask_head, ask_clip);
        }
        if (++asked == kStaged) asked = 0;
        if (ask_half == 0) {
          ask_half = 1;
          return;
        }
        ask_half = 0;
        if (++ask_tile <= 2 * ask_nk) return;
        ask_tile = 0;
        to_ask.next();
        open_step();
      };
      if (one) {
        tma_prefetch_desc(&tmap_q);
        tma_prefetch_desc(&tmap_k);
        tma_prefetch_desc(&tmap_v);
      }
      for (int i = 0; i < kStaged; ++i) ask();
      int slot = 0;
      uint32_t slot_phase = 0;
      const uint32_t src_lane = static_cast<uint32_t>((lane >> 3) * (kD * 4) + (lane & 7) * 32);
      // This warp's half of a tile: eight values a lane and turn, row lane / 8 of four, 16 bytes of the tile's row.
      auto convert = [&](uint8_t* dst, auto type) {
        using T16 = decltype(type);
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          mbar_wait(&sh->staged[c][slot], slot_phase, ctl, status, kErrWaitTma);
          const uint8_t* src = staging + slot * kPieceBytes + src_lane;
          uint8_t* out = dst + (2 * c + half) * (kPieceRows * 128);
          float4 v[kPieceRows / 4][2];
#pragma unroll
          for (int e = 0; e < kPieceRows / 4; ++e) {
            v[e][0] = *reinterpret_cast<const float4*>(src + e * (4 * kD * 4));
            v[e][1] = *reinterpret_cast<const float4*>(src + e * (4 * kD * 4) + 16);
          }
#pragma unroll
          for (int e = 0; e < kPieceRows / 4; ++e)
            *reinterpret_cast<uint4*>(out + sw128_offset(e * 4 + (lane >> 3), lane & 7)) =
                make_uint4(Pack16<T16>::pack(v[e][0].x, v[e][0].y), Pack16<T16>::pack(v[e][0].z, v[e][0].w),
                           Pack16<T16>::pack(v[e][1].x, v[e][1].y), Pack16<T16>::pack(v[e][1].z, v[e][1].w));
          __syncwarp();
          ask();                              // into the piece just read
          if (++slot == kStaged) {
            slot = 0;
            slot_phase ^= 1u;
          }
        }
      };
      auto publish = [&](uint64_t* bar) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
      };
      for (Walk w(shares); w.valid(); w.next()) {
        const int n = w.n, u_lo = w.first() ? w.first_tile_loaded() : w.t;
        // the Q buffer and the slots of the new K tiles, then those of the V tiles, are free: as where TMA fills them
        if (w.first()) {
          if (n >= 1) mbar_wait(&sh->qk_done[(n - 1) & 1], step_phase(n - 1), ctl, status, kErrWaitMma);
        } else if (n >= 2) {
          mbar_wait(&sh->qk_done[n & 1], step_phase(n - 2), ctl, status, kErrWaitMma);
        }
        for (int u = u_lo; u <= w.t; ++u) convert(smem_k + (u & 3) * kTileBytes, __nv_bfloat16());
        convert(smem_q + (n & 1) * kTileBytes, __nv_bfloat16());
        publish(&sh->qk_full[n & 1]);
        if (w.first()) {
          if (n >= 1) mbar_wait(&sh->pv_done[(n - 1) & 1], step_phase(n - 1), ctl, status, kErrWaitMma);
        } else if (w.t - 2 >= w.t0) {
          mbar_wait(&sh->pv_done[n & 1], step_phase(n - 2), ctl, status, kErrWaitMma);
        }
        for (int u = u_lo; u <= w.t; ++u) convert(smem_v + (u & 3) * kTileBytes, VT());
        publish(&sh->v_full[n & 1]);
      }
    } else if (role == 2) {
      // ---------------------------------------------------------- V loads
      if (one) tma_prefetch_desc(&tmap_v);
      for (Walk w(shares); w.valid(); w.next()) {
        const int n = w.n, b = n & 1;
        int u_lo = w.t;
        if (w.first()) {
          // new run: every ring slot may hold a tile of the previous step
          if (n >= 1) mbar_wait(&sh->pv_done[(n - 1) & 1], step_phase(n - 1), ctl, status, kErrWaitMma);
          u_lo = w.first_tile_loaded();
        } else if (w.t - 2 >= w.t0) {
          // the slot held tile t-4, last read by step n-2 of this run
          mbar_wait(&sh->pv_done[b], step_phase(n - 2), ctl, status, kErrWaitMma);
        }
        if (one) {
          mbar_arrive_expect_tx(&sh->v_full[b], static_cast<uint32_t>((w.t - u_lo + 1) * kTileBytes));
          for (int u = u_lo; u <= w.t; ++u)
            tma_load_3d(smem_v + (u & 3) * kTileBytes, &tmap_v, &sh->v_full[b], w.head() * kD, u * kTile, w.clip());
        }
      }
    }
  } else {
    const int kind = warp >> 2;               // the job; 3: results
    const int lg = warp & 3;                  // TMEM lane group
    const int r = lg * 32 + lane;             // row of the tile == TMEM lane
    const uint32_t lanes = static_cast<uint32_t>(lg * 32) << 16;
    if (kind < kJobs) {
      // ---------------------------------------------------------- softmax teams
      const uint32_t job = tmem_base + static_cast<uint32_t>(kind * kTile) + lanes;
      for (Walk w(shares); w.valid(); w.next()) {
        const int n = w.n, x = n & 3;
        const uint32_t xph = static_cast<uint32_t>(n >> 2) & 1u;     // this exchange buffer's use number
        const int w_row0 = w.t * kTile + lg * 32;                    // first frame held by this warp
        const GroupVis vis(w_row0 + lane, w_row0, (w.t - 2 + kind) * kTile, window);

        mbar_wait(&sh->s_full[kind], static_cast<uint32_t>(n) & 1u, ctl, status, kErrWaitMma);
        tc_fence_after_sync();
        float m_raw = tile_row_max(job, vis);                        // -inf for a job with nothing visible
        sh->xm[x][r][kind] = m_raw;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->xm_full[x]);
        mbar_wait(&sh->xm_full[x], xph, ctl, status, kErrWaitConsumer);
        m_raw = fmaxf(fmaxf(sh->xm[x][r][0], sh->xm[x][r][1]), sh->xm[x][r][2]);
        const float m_use = (m_raw == -INFINITY) ? 0.f : m_raw * scale_log2e;
        sh->xl[x][r][kind] = tile_row_probs<VT>(job, job, vis, scale_log2e, m_use);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh->p_full[kind]);
          mbar_arrive(&sh->xl_full[x]);
        }
      }
    } else {
      // ---------------------------------------------------------- results
      for (Walk w(shares); w.valid(); w.next()) {
        const int n = w.n, x = n & 3;
        const int w_row0 = w.t * kTile + lg * 32, i = w_row0 + lane;
        const uint32_t o_addr = tmem_base + kOCol + static_cast<uint32_t>((n & 1) * kD) + lanes;
        mbar_wait(&sh->xl_full[x], static_cast<uint32_t>(n >> 2) & 1u, ctl, status, kErrWaitConsumer);
        const float l_row = sh->xl[x][r][2] + (sh->xl[x][r][0] + sh->xl[x][r][1]);
        mbar_wait(&sh->pv_done[n & 1], step_phase(n), ctl, status, kErrWaitMma);
        tc_fence_after_sync();
        if constexpr (std::is_same<OT, float>::value) {
          uint32_t o[64];
          tmem_ld32(o_addr, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
          tmem_ld32(o_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->o_free[n & 1]);
          if (i < T) {
            const float inv = 1.f / l_row;
            float* dst = out32 + (static_cast<long long>(w.clip()) * T + i) * 512 + w.head() * kD;
#pragma unroll
            for (int d = 0; d < kD; ++d) o[d] = __float_as_uint(__uint_as_float(o[d]) * inv);
#pragma unroll
            for (int d = 0; d < kD; d += 8) st_global_v8(dst + d, o + d);
          }
        } else {
          uint8_t* slab = smem_stage + lg * kSlabBytes;
          if (lane == 0) bulk_wait_group_read<0>();          // the store of the step before has read it
          __syncwarp();
          stage_output_row<VT>(o_addr, slab, lane, 1.f / l_row);
          tc_fence_before_sync();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&sh->o_free[n & 1]);
            if (w_row0 < T) {                                // frames past T are clipped by the map
              tma_store_3d(&tmap_out, slab, w.head() * kD, w_row0, w.clip());
              bulk_commit_group();
            }
          }
        }
      }
      if (lane == 0) bulk_wait_group_read<0>();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);
  if (warp == kSoftmaxWarps) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// q, k, v as FP32 tensors [B, 8, T, 64] of any strides (in values): (64, T, 8, B), boxes of a piece of a tile
static int encode_f32_map(CUtensorMap* map, const void* base, const long long* strides, int B, int T) {
  const cuuint64_t dims[4] = {64, static_cast<cuuint64_t>(T), 8, static_cast<cuuint64_t>(B)};
  const cuuint64_t bytes[3] = {static_cast<cuuint64_t>(strides[2]) * 4, static_cast<cuuint64_t>(strides[1]) * 4,
                               static_cast<cuuint64_t>(B > 1 ? strides[0] : 512) * 4};
  const cuuint32_t box[4] = {64, longclip::kPieceRows, 1, 1}, estr[4] = {1, 1, 1, 1};
  return encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(base), dims, bytes, box, estr, CU_TENSOR_MAP_SWIZZLE_NONE);
}

static int encode_long_map(CUtensorMap* map, const void* base, int B, int T, uint32_t box_rows) {
  // [B, T, 512] 16-bit viewed as (512 fastest, T, B); box = 64 columns x box_rows frames of one clip.
  const cuuint64_t dims[3] = {512, static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(B)};
  const cuuint64_t strides[2] = {512 * 2, static_cast<cuuint64_t>(T) * 512 * 2};
  const cuuint32_t box[3] = {64, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                      CU_TENSOR_MAP_SWIZZLE_128B);
}

// three key tiles per query tile: the window must reach into tile t-2 and not beyond it
bool band_attn_long_takes(int T, int window) {
  return T > 2 * longclip::kTile && window > longclip::kTile + 1 && window <= 2 * longclip::kTile + 1;
}

// The steps of B clips of T frames (at least one) dealt out; false: too many.
static bool long_shares(int B, int T, Shares* shares) {
  const int tiles = (T + longclip::kTile - 1) / longclip::kTile;
  if (static_cast<long long>(B) * 8 * tiles > 0x7fffffffLL) return false;
  *shares = Shares(B * 8, tiles, sm_count());
  return true;
}

int launch_band_attn_long(const void* q, const void* k, const void* v, void* out, int B, int T, int window, float scale,
                          int value_is_fp16, int* status, cudaStream_t st, int dependent, int out_fp32) {
  using namespace longclip;
  if (B <= 0 || !band_attn_long_takes(T, window)) return -1;
  if (out_fp32 && (reinterpret_cast<uintptr_t>(out) & 31u) != 0) return -3;
  CUtensorMap tq, tk, tv, tout;
  int rc = encode_long_map(&tq, q, B, T, kTile);
  if (rc == 0) rc = encode_long_map(&tk, k, B, T, kTile);
  if (rc == 0) rc = encode_long_map(&tv, v, B, T, kTile);     // element size is what matters: 16 bit
  if (rc == 0) rc = out_fp32 ? encode_long_map(&tout, q, B, T, 32) : encode_long_map(&tout, out, B, T, 32);   // FP32: a placeholder
  if (rc != 0) return rc;
  auto kern = out_fp32 ? (value_is_fp16 ? band_attn_long_kernel<__half, float, false> : band_attn_long_kernel<__nv_bfloat16, float, false>)
                       : (value_is_fp16 ? band_attn_long_kernel<__half, __half, false> : band_attn_long_kernel<__nv_bfloat16, __nv_bfloat16, false>);
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes(false));
  if (rc != 0) return rc;
  Shares shares;
  if (!long_shares(B, T, &shares)) return -1;
  return launch_kernel(kern, dim3(shares.used()), threads(false), smem_bytes(false), st, 1, dependent, tq, tk, tv, tout,
                       out_fp32 ? static_cast<float*>(out) : nullptr, shares, T, window, scale * 1.4426950408889634f, status);
}

// Strides that a tensor map can have, and enough steps a block.  The converting warps keep up with the chain of steps, but where a
// run begins the first step waits until they have made seven tiles instead of three, and a short call is little else; a converting
// pass in front costs 1 us and 0.7 ns a frame.  Inside from four steps on, from six where short sequences begin and end inside of shares.
// GPU time, FP32, in front -> inside (350 calls of 1 to 12 steps: what goes inside is 4 % slower there at most, what does not 9 % slower in front):
//   1 or 2 steps   1 clip of 257 frames 8.7 -> 11.0 us, 1 of 2500 14.9 -> 17.1, 8 of 300 14.0 -> 14.2
//   3              18 of 257 18.2 -> 18.2, 9 of 513 19.2 -> 19.7, 6 of 900 21.9 -> 23.0
//   4              16 of 385 23.3 -> 22.5, 7 of 900 24.4 -> 25.4, 9 of 1000 30.9 -> 28.4, 6 of 1500 31.4 -> 27.5, 3 of 2500 28.3 -> 27.0; shares
//                  run on: 12 of 700 29.5 -> 27.3, but 24 of 257 23.9 -> 27.1, 12 of 513 24.3 -> 26.1
//   5              18 of 513 32.5 -> 27.3, 15 of 700 37.2 -> 32.4; run on: 25 of 257 26.3 -> 29.4, 28 of 300 30.4 -> 30.4, 23 of 385 32.3 -> 31.9
//   6              37 of 257 35.1 -> 30.9; run on: 24 of 385 35.6 -> 34.8, 22 of 513 41.2 -> 37.4
//   7 and more     41 of 257 41.0 -> 39.9, 19 of 700 49.0 -> 41.9, 18 of 900 57.9 -> 44.0, 11 of 2500 91.7 -> 65.7
bool band_attn_long_takes_f32(const long long* strides, int B, int T) {
  for (int i = 0; i < 9; ++i) {
    if (i % 3 == 0 && B == 1) continue;
    if (strides[i] < 4 || strides[i] % 4 != 0 || strides[i] >= (1ll << 38)) return false;
  }
  Shares s;
  if (!long_shares(B, T, &s)) return false;
  const bool run_on = s.cuts == 0 && s.per_block % s.tiles != 0;
  return s.per_block >= (run_on && s.tiles <= 5 ? 6 : 4);
}

int launch_band_attn_long_f32(const void* const* qkv, const long long* strides, float* out, int B, int T, int window, float scale,
                              int value_is_fp16, int* status, cudaStream_t st) {
  using namespace longclip;
  if (B <= 0 || !band_attn_long_takes(T, window) || !band_attn_long_takes_f32(strides, B, T)) return -1;
  if ((reinterpret_cast<uintptr_t>(out) & 31u) != 0) return -3;
  CUtensorMap maps[4];
  int rc = 0;
  for (int i = 0; i < 3 && rc == 0; ++i) {
    if ((reinterpret_cast<uintptr_t>(qkv[i]) & 15u) != 0) return -3;
    rc = encode_f32_map(&maps[i], qkv[i], strides + 3 * i, B, T);
  }
  if (rc != 0) return rc;
  maps[3] = maps[0];                                   // a placeholder: FP32 rows are stored from registers
  auto kern = value_is_fp16 ? band_attn_long_kernel<__half, float, true> : band_attn_long_kernel<__nv_bfloat16, float, true>;
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes(true));
  if (rc != 0) return rc;
  Shares shares;
  if (!long_shares(B, T, &shares)) return -1;
  return launch_kernel(kern, dim3(shares.used()), threads(true), smem_bytes(true), st, 1, 0, maps[0], maps[1], maps[2], maps[3], out, shares, T,
                       window, scale * 1.4426950408889634f, status);
}

}  // namespace fm
