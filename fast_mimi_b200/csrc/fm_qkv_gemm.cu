// QKV projection with a RoPE epilogue for sm_100a.
//
//   [q | k | v][m, :] = x[m, :] * W_qkv^T          (M frames x 1536 outputs x K=512, BF16 in, FP32 acc)
//   q, k <- rotate-half RoPE at the frame's position  (FP32, before rounding to 16 bit)
//
// Replaces the three bias-free projections plus _apply_rope of the reference
// (src/fast_mimi/model.py:1897-1912; packed form src/fast_mimi/_packed_qkv.py:139-171).
//
// Two CTAs on neighbouring SMs work as a pair (cluster of 2, tcgen05 cta_group::2).  Each CTA owns a
// 128-frame tile of x, loaded once by TMA and kept in shared memory (128 KB), and loads HALF of every
// 256x64 W_qkv tile (128 weight rows); one tcgen05.mma issued by the pair's leader multiplies the
// 256 frames of both CTAs by all 256 weight rows, so each W byte is fetched from L2 once per 256 frames.
// Each CTA's 128x256 FP32 result lands in its own TMEM (two 256-column buffers: the epilogue of one work
// unit overlaps the MMAs of the next).  The kernel is persistent: 74 pairs walk contiguous ranges of
// (frame-tile pair, output tile) units, and while the last output tile of a frame tile is being multiplied
// the x chunks it has finished with are already replaced by the next frame tile's.  Epilogue warps read one
// frame row per thread (both halves of a RoPE pair sit in the same row), hand the accumulator back as soon
// as their last tensor-memory load has completed, rotate, round, stage 32x64 slabs in swizzled shared memory
// and write them with TMA stores (full 128-byte lines).  Warps 0-7: epilogue (two per TMEM lane group, two
// heads each).  Warp 8: W producer (+ TMEM allocation).  Warp 9: MMA issuer (leader CTA only).  Warp 10:
// x producer.
#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"

namespace fm {

namespace gemm {
constexpr int kBlockM = 128;           // frames per CTA
constexpr int kBlockN = 256;           // outputs per tile (4 heads of q, k or v)
constexpr int kHalfN = kBlockN / 2;    // weight rows loaded by each CTA of the pair
constexpr int kBlockK = 64;            // one 128-byte swizzle row of BF16
constexpr int kHidden = 512;           // K
constexpr int kKChunks = kHidden / kBlockK;
constexpr int kStages = 4;
constexpr int kABytes = kBlockM * kBlockK * 2;   // 16 KB per K chunk
constexpr int kBBytes = kHalfN * kBlockK * 2;    // 16 KB per stage per CTA
constexpr int kSlabBytes = 32 * 128;             // one warp's 32 frames x 64 outputs x 16 bit
constexpr int kEpiWarps = 8;                     // two per TMEM lane group: heads 0,1 and heads 2,3 of a tile
constexpr int kHeadsPerWarp = 16 / kEpiWarps;    // a tile has four heads per lane group
constexpr int kThreads = (kEpiWarps + 3) * 32;   // + W producer, MMA issuer, x producer
constexpr int kTmemCols = 512;
constexpr int kSmemBytes = 1024 /*align*/ + kKChunks * kABytes + kStages * kBBytes + kEpiWarps * kSlabBytes + 256;

struct Barriers {
  uint64_t a_full[kKChunks];   // used in the leader: bytes of both CTAs' x chunks
  uint64_t a_empty[kKChunks];  // per CTA: the chunk's last MMA of the current frame tile has completed
  uint64_t b_full[kStages];    // used in the leader: bytes of both halves of a W tile
  uint64_t b_empty[kStages];   // per CTA: stage consumed by the tensor core
  uint64_t acc_full[2];        // per CTA: accumulator buffer complete
  uint64_t acc_empty[2];       // used in the leader: 16 epilogue warps (8 per CTA) drained the buffer
  uint32_t tmem_base;
  uint32_t skip;               // leader's view of "status already non-zero at start"
  CtaCtl ctl;
};
static_assert(sizeof(Barriers) <= 256, "barrier block too large");
}  // namespace gemm

template <typename VT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm::kThreads, 1)
qkv_rope_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                     const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, QkvEpilogueArgs ep, int M, int total_units,
                     uint32_t idesc, int* status) {
  using namespace gemm;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;                                   // kKChunks x [128 rows x 128 B]
  uint8_t* smem_b = smem_a + kKChunks * kABytes;            // kStages  x [128 rows x 128 B]
  uint8_t* smem_out = smem_b + kStages * kBBytes;           // kEpiWarps x [32 rows x 128 B]
  Barriers* bars = reinterpret_cast<Barriers*>(smem_out + kEpiWarps * kSlabBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();      // 0 = pair leader
  const bool leader = rank == 0;
  // Work units = (pair of 128-frame tiles, 256-wide output tile), numbered frame-tile-major, so that a
  // pair walks the six output tiles of one frame tile before moving to the next.  Each pair takes a
  // contiguous range of units.
  const int pair = static_cast<int>(blockIdx.x >> 1), n_pairs = static_cast<int>(gridDim.x >> 1);
  const int u_base = total_units / n_pairs, u_extra = total_units % n_pairs;
  const int u_begin = pair * u_base + (pair < u_extra ? pair : u_extra);
  const int u_count = u_base + (pair < u_extra ? 1 : 0);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kKChunks; ++i) {
      mbar_init(&bars->a_full[i], 1);
      mbar_init(&bars->a_empty[i], 1);
    }
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->b_full[i], 1);
      mbar_init(&bars->b_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], 2 * kEpiWarps);
    }
    bars->ctl.abort = 0;
    bars->skip = (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0) ? 1u : 0u;
    fence_mbar_init();
  }
  if (warp == kEpiWarps) {
    tmem_alloc_pair(&bars->tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();            // both CTAs' barriers exist before anything signals across the pair
  griddep_launch();
  if (warp != kEpiWarps) griddep_wait();   // x may come from the kernel in front; the W loads need not wait for it
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  CtaCtl* ctl = &bars->ctl;
  // Both CTAs take the leader's decision, so the pair stays in step.
  const bool skip = ld_shared_cluster_u32(map_to_cta(smem_u32(&bars->skip), 0)) != 0;

  if (skip) {
    // a previous kernel already reported a timeout through this status word: do nothing
  } else if (warp == kEpiWarps) {
    // ------------------------------------------------------------ W producer (one thread per CTA)
    if (lane == 0) {
      tma_prefetch_desc(&tmap_w);
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < u_count; ++i) {
        const int ntile = (u_begin + i) % ep.n_tiles;
        const int n0 = ntile * kBlockN + static_cast<int>(rank) * kHalfN;
        for (int kc = 0; kc < kKChunks; ++kc) {
          mbar_wait(&bars->b_empty[stage], phase ^ 1u, ctl, status, kErrWaitConsumer);
          if (leader) mbar_arrive_expect_tx(&bars->b_full[stage], 2 * kBBytes);
          tma_load_2d_pair(smem_b + stage * kBBytes, &tmap_w, &bars->b_full[stage], kc * kBlockK, n0);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == kEpiWarps + 2) {
    // ------------------------------------------------------------ x producer (one thread per CTA)
    // Runs on its own so that waiting for a chunk's last MMA never holds up the W stream: each chunk of
    // the resident x tile is replaced by the next frame tile's as soon as the tensor core is done with it.
    if (lane == 0) {
      tma_prefetch_desc(&tmap_x);
      int gen = -1, cur_tile = -1;
      for (int i = 0; i < u_count; ++i) {
        const int frame_tile = (u_begin + i) / ep.n_tiles;
        if (frame_tile == cur_tile) continue;
        cur_tile = frame_tile;
        ++gen;
        for (int kc = 0; kc < kKChunks; ++kc) {
          if (gen > 0) mbar_wait(&bars->a_empty[kc], static_cast<uint32_t>(gen - 1) & 1u, ctl, status, kErrWaitMma);
          if (leader) mbar_arrive_expect_tx(&bars->a_full[kc], 2 * kABytes);
          tma_load_2d_pair(smem_a + kc * kABytes, &tmap_x, &bars->a_full[kc], kc * kBlockK,
                           (2 * frame_tile + static_cast<int>(rank)) * kBlockM);
        }
      }
    }
  } else if (warp == kEpiWarps + 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    // The whole warp walks the loop and one elected lane issues: with warp-uniform control flow the descriptors
    // stay in uniform registers, and the per-chunk wait / four MMAs / commit sequence keeps the tensor core fed
    // (128 cycles per MMA in isolation against 195 when a single lane runs the same loop under a lane test).
    if (leader) {
      const bool elected = elect_one();
      int stage = 0, gen = -1, cur_tile = -1;
      uint32_t phase = 0;
      for (int i = 0; i < u_count; ++i) {
        const int u = u_begin + i, frame_tile = u / ep.n_tiles;
        const bool fresh = frame_tile != cur_tile;        // first unit of a frame tile: wait for its x chunks
        if (fresh) { ++gen; cur_tile = frame_tile; }
        const int next_tile = (i + 1 < u_count) ? (u + 1) / ep.n_tiles : -1;
        const bool roll = next_tile >= 0 && next_tile != frame_tile;
        const int buf = i & 1;
        const uint32_t use = static_cast<uint32_t>(i >> 1);
        mbar_wait(&bars->acc_empty[buf], (use & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * kBlockN);
        for (int kc = 0; kc < kKChunks; ++kc) {
          if (fresh) mbar_wait(&bars->a_full[kc], static_cast<uint32_t>(gen) & 1u, ctl, status, kErrWaitTma);
          mbar_wait(&bars->b_full[stage], phase, ctl, status, kErrWaitTma);
          tc_fence_after_sync();
          const uint64_t a_desc = umma_desc_sw128(smem_u32(smem_a + kc * kABytes));
          const uint64_t b_desc = umma_desc_sw128(smem_u32(smem_b + stage * kBBytes));
#pragma unroll
          for (int ks = 0; ks < kBlockK / 16; ++ks) {
            // +32 bytes per 16-element K step inside the 128-byte swizzle row (encoded >> 4).
            if (elected) tc_mma_ss_pair(d_tmem, a_desc + 2u * ks, b_desc + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
          }
          if (elected) {
            tc_commit_pair(&bars->b_empty[stage], 3);     // frees the stage in both CTAs
            if (roll) tc_commit_pair(&bars->a_empty[kc], 3);   // and, on a tile's last unit, the x chunk
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (elected) tc_commit_pair(&bars->acc_full[buf], 3);        // both CTAs' epilogues may read their TMEM
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 0..7 of both CTAs)
    const int lg = warp & 3;      // TMEM lane group: frames 32*lg .. 32*lg+31 of the tile
    const int hsel = warp >> 2;   // which two of the tile's four heads this warp handles
    const int row_in_tile = lg * 32 + lane;
    const uint32_t acc_empty_leader = map_to_cta(smem_u32(&bars->acc_empty[0]), 0);
    uint8_t* slab = smem_out + warp * kSlabBytes;
    // Per frame tile: this thread's frame, its RoPE factors (kept in registers for all heads of q and k;
    // the table's two 32-wide halves are identical by construction, so only the first is read) and its
    // ring slot.
    float rc[32], rs[32];
    long long row = 0, ring_row = -1;
    bool row_ok = false;
    int m0 = 0, cur_tile = -1;
    for (int i = 0; i < u_count; ++i) {
      const int u = u_begin + i, frame_tile = u / ep.n_tiles, ntile = u % ep.n_tiles;
      if (frame_tile != cur_tile) {
        cur_tile = frame_tile;
        m0 = (2 * frame_tile + static_cast<int>(rank)) * kBlockM;
        row = static_cast<long long>(m0) + row_in_tile;
        row_ok = row < M;
        const int clip = row_ok ? static_cast<int>(row / ep.T) : 0;
        const int t = row_ok ? static_cast<int>(row % ep.T) : 0;
        if (row_ok && ep.cos != nullptr) {
          const float4* c4 = reinterpret_cast<const float4*>(ep.cos + clip * ep.cos_bstride + static_cast<long long>(t) * 64);
          const float4* s4 = reinterpret_cast<const float4*>(ep.sin + clip * ep.cos_bstride + static_cast<long long>(t) * 64);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 c = __ldg(c4 + j), sn = __ldg(s4 + j);
            rc[4 * j] = c.x; rc[4 * j + 1] = c.y; rc[4 * j + 2] = c.z; rc[4 * j + 3] = c.w;
            rs[4 * j] = sn.x; rs[4 * j + 1] = sn.y; rs[4 * j + 2] = sn.z; rs[4 * j + 3] = sn.w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) { rc[j] = 1.f; rs[j] = 0.f; }
        }
        ring_row = -1;
        if (ep.ring_k != nullptr && row_ok) {
          const int pos = ep.pos_base + (ep.clip_pos != nullptr ? ep.clip_pos[clip] : 0) + t;
          // Only the newest ring_slots frames of a clip land in the ring.  A negative position would index
          // another stream's ring: it is recorded and the write is dropped.
          if (pos < 0) {
            if (status != nullptr) atomicMax(status, static_cast<int>(kErrBounds));
          } else if (t >= ep.T - ep.ring_slots) {
            ring_row = static_cast<long long>(clip) * 8 * ep.ring_slots + pos % ep.ring_slots;
          }
        }
      }
      const int buf = i & 1;
      const uint32_t use = static_cast<uint32_t>(i >> 1);
      const int seg = ep.seg_base + (ntile >> 1);   // 0 = q, 1 = k, 2 = v or the plain output
      mbar_wait(&bars->acc_full[buf], use & 1u, ctl, status, kErrWaitMma);
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + static_cast<uint32_t>(buf * kBlockN);
      const CUtensorMap* omap = seg == 0 ? &tmap_q : (seg == 1 ? &tmap_k : &tmap_v);
      const bool lin_ok = (seg == 0 ? ep.q : (seg == 1 ? ep.k : ep.v)) != nullptr;
      uint16_t* ring = seg == 1 ? ep.ring_k : (seg == 2 ? ep.ring_v : nullptr);
#pragma unroll 1
      for (int hh = hsel * kHeadsPerWarp; hh < (hsel + 1) * kHeadsPerWarp; ++hh) {
        const int head = (ntile & 1) * 4 + hh;
        if (lin_ok) {
          // The previous store out of this warp's slab must have finished reading it.
          if (lane == 0) bulk_wait_group_read<0>();
          __syncwarp();
        }
        uint4* ring_dst = (ring != nullptr && ring_row >= 0)
                              ? reinterpret_cast<uint4*>(ring + (ring_row + static_cast<long long>(head) * ep.ring_slots) * 64)
                              : nullptr;
#pragma unroll
        for (int piece = 0; piece < 2; ++piece) {
          // 16 columns of the head's first half and the 16 columns 32 further on: a RoPE pair set.
          uint32_t lo[16], hi[16];
          tmem_ld16(t_row + hh * 64 + piece * 16, lo);
          tmem_ld16(t_row + hh * 64 + 32 + piece * 16, hi);
          tmem_ld_wait();
          if (hh == (hsel + 1) * kHeadsPerWarp - 1 && piece == 1) {
            // That was this warp's last read of the accumulator: hand it back before the arithmetic and the
            // stores.  The loads have completed, so the arrival needs no release ordering.
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty_leader + static_cast<uint32_t>(buf) * 8u);
          }
          uint32_t plo[8], phi[8];
          if (seg < 2) {
#pragma unroll
            for (int d = 0; d < 16; d += 2) {
              float o_lo[2], o_hi[2];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float a = __uint_as_float(lo[d + e]), b = __uint_as_float(hi[d + e]);
                const float c = rc[piece * 16 + d + e], sn = rs[piece * 16 + d + e];
                o_lo[e] = a * c - b * sn;
                o_hi[e] = b * c + a * sn;
              }
              plo[d / 2] = Pack16<__nv_bfloat16>::pack(o_lo[0], o_lo[1]);
              phi[d / 2] = Pack16<__nv_bfloat16>::pack(o_hi[0], o_hi[1]);
            }
          } else {
            if (ep.out_scale != nullptr) {
              // per-channel factor: the same address in every lane, so one broadcast load each
              const float4* s_lo = reinterpret_cast<const float4*>(ep.out_scale + head * 64 + piece * 16);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float4 a = __ldg(s_lo + j), b = __ldg(s_lo + 8 + j);
                lo[4 * j] = __float_as_uint(__uint_as_float(lo[4 * j]) * a.x);
                lo[4 * j + 1] = __float_as_uint(__uint_as_float(lo[4 * j + 1]) * a.y);
                lo[4 * j + 2] = __float_as_uint(__uint_as_float(lo[4 * j + 2]) * a.z);
                lo[4 * j + 3] = __float_as_uint(__uint_as_float(lo[4 * j + 3]) * a.w);
                hi[4 * j] = __float_as_uint(__uint_as_float(hi[4 * j]) * b.x);
                hi[4 * j + 1] = __float_as_uint(__uint_as_float(hi[4 * j + 1]) * b.y);
                hi[4 * j + 2] = __float_as_uint(__uint_as_float(hi[4 * j + 2]) * b.z);
                hi[4 * j + 3] = __float_as_uint(__uint_as_float(hi[4 * j + 3]) * b.w);
              }
            }
            if (ep.resid != nullptr && row_ok) {
              // this frame's 32 + 32 bytes of the residual: whole sectors, read once
              const uint4* r_lo = reinterpret_cast<const uint4*>(ep.resid + row * 512 + head * 64 + piece * 16);
              const uint4 r[4] = {r_lo[0], r_lo[1], r_lo[4], r_lo[5]};
              const uint32_t* rw = reinterpret_cast<const uint32_t*>(r);
#pragma unroll
              for (int d = 0; d < 16; d += 2) {
                const float2 a = Pack16<VT>::unpack(rw[d / 2]), b = Pack16<VT>::unpack(rw[8 + d / 2]);
                lo[d] = __float_as_uint(__uint_as_float(lo[d]) + a.x);
                lo[d + 1] = __float_as_uint(__uint_as_float(lo[d + 1]) + a.y);
                hi[d] = __float_as_uint(__uint_as_float(hi[d]) + b.x);
                hi[d + 1] = __float_as_uint(__uint_as_float(hi[d + 1]) + b.y);
              }
            }
#pragma unroll
            for (int d = 0; d < 16; d += 2) {
              plo[d / 2] = Pack16<VT>::pack(__uint_as_float(lo[d]), __uint_as_float(lo[d + 1]));
              phi[d / 2] = Pack16<VT>::pack(__uint_as_float(hi[d]), __uint_as_float(hi[d + 1]));
            }
          }
          if (lin_ok) {
            // Row `lane` of the slab, 16-byte chunks 2p, 2p+1 (first half) and 4+2p, 4+2p+1 (second half).
            *reinterpret_cast<uint4*>(slab + sw128_offset(lane, piece * 2)) = make_uint4(plo[0], plo[1], plo[2], plo[3]);
            *reinterpret_cast<uint4*>(slab + sw128_offset(lane, piece * 2 + 1)) = make_uint4(plo[4], plo[5], plo[6], plo[7]);
            *reinterpret_cast<uint4*>(slab + sw128_offset(lane, 4 + piece * 2)) = make_uint4(phi[0], phi[1], phi[2], phi[3]);
            *reinterpret_cast<uint4*>(slab + sw128_offset(lane, 4 + piece * 2 + 1)) = make_uint4(phi[4], phi[5], phi[6], phi[7]);
          }
          if (ring_dst != nullptr) {
            ring_dst[piece * 2] = make_uint4(plo[0], plo[1], plo[2], plo[3]);
            ring_dst[piece * 2 + 1] = make_uint4(plo[4], plo[5], plo[6], plo[7]);
            ring_dst[4 + piece * 2] = make_uint4(phi[0], phi[1], phi[2], phi[3]);
            ring_dst[4 + piece * 2 + 1] = make_uint4(phi[4], phi[5], phi[6], phi[7]);
          }
        }
        if (lin_ok) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            // Rows past M are clipped by the tensor map.
            tma_store_2d(omap, slab, head * 64, m0 + lg * 32);
            bulk_commit_group();
          }
        }
      }
    }
    if (lane == 0) bulk_wait_group_read<0>();
  }

  // Teardown: neither CTA may leave (or release TMEM) while its partner can still signal it.
  tc_fence_before_sync();
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);   // copies that may still be in flight get time to land
  cluster_sync_all();
  if (warp == kEpiWarps) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

static int launch_gemm(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags,
                       int* status, cudaStream_t st, int dependent) {
  using namespace gemm;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_qkv) | reinterpret_cast<uintptr_t>(ep.q) |
       reinterpret_cast<uintptr_t>(ep.k) | reinterpret_cast<uintptr_t>(ep.v) | reinterpret_cast<uintptr_t>(ep.ring_k) |
       reinterpret_cast<uintptr_t>(ep.ring_v)) & 15u)
    return -3;
  CUtensorMap tmap_x, tmap_w, tmap_q, tmap_k, tmap_v;
  int rc = encode_rows_16bit(&tmap_x, x, static_cast<uint64_t>(M), kHidden, kBlockM, kBlockK);
  if (rc != 0) return rc;
  rc = encode_rows_16bit(&tmap_w, w_qkv, static_cast<uint64_t>(ep.n_tiles) * kBlockN, kHidden, kHalfN, kBlockK);
  if (rc != 0) return rc;
  // Output maps (16-bit elements whatever the float format); a missing output reuses x as a placeholder
  // that the kernel never stores through.
  rc = encode_rows_16bit(&tmap_q, ep.q != nullptr ? ep.q : x, static_cast<uint64_t>(M), 512, 32, 64);
  if (rc != 0) return rc;
  rc = encode_rows_16bit(&tmap_k, ep.k != nullptr ? ep.k : x, static_cast<uint64_t>(M), 512, 32, 64);
  if (rc != 0) return rc;
  rc = encode_rows_16bit(&tmap_v, ep.v != nullptr ? ep.v : x, static_cast<uint64_t>(M), 512, 32, 64);
  if (rc != 0) return rc;
  const int m_tiles = (M + kBlockM - 1) / kBlockM;
  const int pair_tiles = (m_tiles + 1) / 2;          // an odd last tile gets a partner that works on padding
  const int total_units = pair_tiles * ep.n_tiles;            // (pair of frame tiles, 256-wide output tile)
  const int max_pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;   // persistent: one CTA per SM, CTAs in pairs
  const int n_pairs = total_units < max_pairs ? total_units : max_pairs;
  // dtype_flags bit 0: v is written as FP16 (else BF16); bit 1: x and w_qkv hold FP16 (else BF16).
  const int in_fmt = (dtype_flags & 2) ? 0 : 1;   // tcgen05 kind::f16 operand format: 0 = F16, 1 = BF16
  const uint32_t idesc = umma_idesc_f16(2 * kBlockM, kBlockN, in_fmt, in_fmt, 0, 0);
  auto kern = (dtype_flags & 1) ? qkv_rope_gemm_kernel<__half> : qkv_rope_gemm_kernel<__nv_bfloat16>;
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes);
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(2 * n_pairs), kThreads, kSmemBytes, st, 1, dependent, tmap_x, tmap_w, tmap_q, tmap_k, tmap_v,
                       ep, M, total_units, idesc, status);
}

int launch_qkv_rope_gemm(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep_in, int M, int dtype_flags,
                         int* status, cudaStream_t st, int dependent) {
  if (M <= 0) return M == 0 ? 0 : -1;
  if (ep_in.T <= 0 || absent(x, w_qkv, ep_in.cos, ep_in.sin)) return -1;
  if (!rope_tables_aligned(ep_in.cos, ep_in.sin, ep_in.cos_bstride)) return -3;
  QkvEpilogueArgs ep = ep_in;
  ep.n_tiles = 6;
  ep.seg_base = 0;
  ep.out_scale = nullptr;
  ep.resid = nullptr;
  if (few_row_tiles(M, 1536)) {
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_qkv) | reinterpret_cast<uintptr_t>(ep.q) |
         reinterpret_cast<uintptr_t>(ep.k) | reinterpret_cast<uintptr_t>(ep.v) | reinterpret_cast<uintptr_t>(ep.ring_k) |
         reinterpret_cast<uintptr_t>(ep.ring_v)) & 15u)
      return -3;
    // weights resident in tensor memory, by itself to 768 rows (the few-row kernel -> that one, us: 1 row 5.4 -> 4.7, 64 5.9 -> 5.0, 125 7.0 -> 5.3, 250 7.9 -> 5.5, 768
    // 7.9 -> 7.1), in a chain to 1024 (eight layers of 8 clips of 125 frames 307 -> 304, 4 of 250 BF16 frames 318 -> 312, 1024 live streams 912 -> 909)
    if (linear_ws_takes(M, 1536, 512, dependent)) return launch_qkv_ws(x, w_qkv, ep, M, dtype_flags, status, st, dependent);
    return launch_qkv_small(x, w_qkv, ep, M, dtype_flags, status, st, dependent);
  }
  return launch_gemm(x, w_qkv, ep, M, dtype_flags, status, st, dependent);
}

int launch_out_proj_gemm(const void* a, const void* w, void* y, const float* out_scale, const void* resid, int M,
                         int dtype_flags, int* status, cudaStream_t st) {
  if (M <= 0) return M == 0 ? 0 : -1;
  if (a == nullptr || w == nullptr || y == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(out_scale) | reinterpret_cast<uintptr_t>(resid)) & 15u) return -3;
  QkvEpilogueArgs ep = {};
  ep.v = static_cast<uint16_t*>(y);
  ep.T = M;             // one "clip": positions are not used without RoPE
  ep.ring_slots = 1;
  ep.n_tiles = 2;
  ep.seg_base = 2;
  ep.out_scale = out_scale;
  ep.resid = static_cast<const uint16_t*>(resid);
  return launch_gemm(a, w, ep, M, dtype_flags, status, st, 0);
}

}  // namespace fm
