// General bias-free linear layer for sm_100a with a fused epilogue:
//
//   y[m, :] = residual[m, :] + scale * act(a[m, :] * W^T)      (M rows x N outputs x K inputs, 16-bit in, FP32 acc)
//
// act is the identity or the exact (erf) GELU; scale (per output channel) and residual are optional; y and
// the residual are BF16, FP16 or FP32.  It serves the linear layers that follow the attention core in the
// reference's transformer layer: the MLP  fc2(gelu(fc1(.)))  with its layer scale and residual add
// (src/fast_mimi/model.py:1990-1999, :2060-2061) and, with FP32 residual streams, the output projection
// (src/fast_mimi/model.py:1961, :2059).
//
// Unlike the QKV projection kernel, which keeps its x tile resident because K is only 512, both operands
// stream here: a stage holds a 128 x 64 slice of a and a 128 x 64 slice of W per CTA (32 KB), five or six stages deep.
// Two CTAs form a pair (cluster of 2, tcgen05 cta_group::2): one tcgen05.mma multiplies the pair's 256 rows by
// 256 (or 128) weight rows, each CTA contributing half of the weight tile.  Accumulators: two 256-column TMEM buffers
// per CTA, so the epilogue of one unit overlaps the MMAs of the next.  Persistent: (row-tile pair, 256-wide
// output tile) units, numbered row-tile-major, are dealt round-robin to the pairs, so the output tiles of a
// row tile are computed at the same time by neighbouring pairs and share its a slices through L2.
// Two shapes of the same kernel (template parameter kWide):
//   wide    warps 0-15 epilogue (four per TMEM lane group, one 64-column group of the unit each), warp 16 TMA
//           producer (+ TMEM allocation), warp 17 MMA issuer (leader CTA only); five stages.  For epilogues that
//           carry arithmetic (the exact GELU, the candidate records of the quantiser search): there the epilogue,
//           not the tensor core, bounds the kernel, and eight warps cannot hide its latencies.  Five warps per SM
//           sub-partition leave 96 registers per thread at launch; the load / issue warpgroup shrinks to 32 and the
//           epilogue warpgroups grow to 112 (setmaxnreg: 512 x 112 + 128 x 32 = 640 x 96).
//   narrow  warps 0-7 epilogue (two 64-column groups each, one with 128-wide units), warps 8 and 9 producer and issuer;
//           six (seven) stages (the shared memory of eight staging slabs buys the sixth, which the K = 2048 layer uses).
#include <type_traits>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"

namespace fm {

namespace lin {
constexpr int kBlockM = 128;           // rows per CTA
constexpr int kBlockK = 64;            // one 128-byte swizzle row of 16-bit values
constexpr int kABytes = kBlockM * kBlockK * 2;   // 16 KB
constexpr int kSlabBytes = 32 * 128;             // one warp's staging: 32 rows x 128 bytes
template <bool kWide, int kBlockN> struct Shape {
  static constexpr int kHalfN = kBlockN / 2;              // weight rows loaded by each CTA of the pair
  static constexpr int kStageBytes = kABytes + kHalfN * kBlockK * 2;
  static constexpr int kStages = kWide ? 5 : (kBlockN == 256 ? 6 : 7);
  static constexpr int kEpiWarps = kWide ? 16 : 8;
  static constexpr int kGroupsPerWarp = kBlockN / 16 / kEpiWarps;   // a unit has kBlockN / 64 64-column groups per lane group
  static constexpr int kTmemCols = 2 * kBlockN;
  // wide: five warpgroups, the last one holds the producer and the issuer; narrow: epilogue warps + 2
  static constexpr int kThreads = kWide ? (kEpiWarps + 4) * 32 : (kEpiWarps + 2) * 32;
  static constexpr int kSmemBytes = 1024 /*align*/ + kStages * kStageBytes + kEpiWarps * kSlabBytes + 256;
};
constexpr int kEpiRegs = 112, kIssueRegs = 32;
static_assert(512 * kEpiRegs + 128 * kIssueRegs <= Shape<true, 256>::kThreads * 96, "register pool of the launch");

struct Barriers {
  uint64_t full[7];            // used in the leader: bytes of both CTAs' a and W slices
  uint64_t empty[7];           // per CTA: stage consumed by the tensor core
  uint64_t acc_full[2];        // per CTA: accumulator buffer complete
  uint64_t acc_empty[2];       // used in the leader: the epilogue warps of both CTAs drained the buffer
  uint32_t tmem_base;
  uint32_t skip;
  CtaCtl ctl;
};
static_assert(sizeof(Barriers) <= 256, "barrier block too large");

}  // namespace lin

struct LinearArgs {
  ParamVec scale;         // [N] or null             (kOut 3: |e_j|^2 of the codebook entries, FP32)
  const void* resid;      // [M, N] in the output's type or null      (kOut 3: per-row candidate margin, [M] FP32)
  int M, N, K;
  int gelu;               // 1: exact GELU on the accumulator before scale / residual
  uint4* records;         // kOut 3: [M, N / 64] candidate records
  void* y;                // [M, N]: stored directly where there is a residual, through the tensor map otherwise
  SplitRows rows;         // kOut 4
};

// kOut: 0 = BF16, 1 = FP16, 2 = FP32 (type of y and of the residual); 3 = no y at all: the products are the inner
// products x . e_j of a nearest-entry search and the epilogue reduces every 64 of them to one 16-byte record
// {min_j d_j, 64-bit mask of the entries with d_j <= min + margin[row]},  d_j = |e_j|^2 - 2 x . e_j  (see fm_rvq.cu).
// 4 = FP32 y of a split-precision product: both operands are pairs of FP16 matrices hi + lo, and K runs three times,
// lo W_hi, hi W_lo, hi W_hi (the small terms first), into one accumulator (or, for two products that are to be added, into one
// each).  As three products that handed FP32 sums on
// through memory the same work moved 20 bytes per output value instead of four (64000 rows, K = 2048, N = 512: 317 us here,
// 1.27 PFLOP/s over the three terms).
template <int kOut, bool kWide, int kBlockN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(lin::Shape<kWide, kBlockN>::kThreads, 1)
linear_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ SplitMaps<kOut == 4> low,
                   const __grid_constant__ LinearArgs args, int total_units,
                   uint32_t idesc, int* status) {
  using namespace lin;
  constexpr bool kSplit = kOut == 4, kF32 = kOut == 2 || kOut == 4;
  using S = Shape<kWide, kBlockN>;
  constexpr int kStages = S::kStages, kEpiWarps = S::kEpiWarps, kGroupsPerWarp = S::kGroupsPerWarp;
  constexpr int kStageBytes = S::kStageBytes, kHalfN = S::kHalfN, kTmemCols = S::kTmemCols;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_stage = smem;                                  // kStages x [a slice | W slice]
  uint8_t* smem_out = smem_stage + kStages * kStageBytes;      // kEpiWarps x 4 KB
  Barriers* bars = reinterpret_cast<Barriers*>(smem_out + kEpiWarps * kSlabBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = rank == 0;
  const int n_tiles = args.N / kBlockN;
  const int k_chunks = (kSplit ? 3 : 1) * (args.K / kBlockK);
  // accumulators per unit (a split-precision product of two parts fills both buffers), K chunks of one
  const int n_acc = kSplit ? args.rows.parts : 1, part_chunks = args.K / kBlockK / n_acc, acc_chunks = k_chunks / n_acc;
  // Units are dealt round-robin: at any moment neighbouring pairs work on the output tiles of the SAME rows,
  // so the slices of a that one of them pulls from HBM are L2 hits for the others (with contiguous ranges
  // per pair the second output tile of a row tile came 30 us after the first and its a tile had been evicted:
  // 1.85x the algorithmic reads for K = 2048).
  const int pair = static_cast<int>(blockIdx.x >> 1), n_pairs = static_cast<int>(gridDim.x >> 1);
  const int u_count = (total_units - pair + n_pairs - 1) / n_pairs;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
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
  cluster_sync_all();
  griddep_launch();
  if (warp != kEpiWarps) griddep_wait();   // the residual may come from the kernel in front (the producer waits below)
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  CtaCtl* ctl = &bars->ctl;
  const bool skip = ld_shared_cluster_u32(map_to_cta(smem_u32(&bars->skip), 0)) != 0;

  if (skip) {
    // a previous kernel already reported a timeout through this status word: do nothing
  } else if (warp >= kEpiWarps) {
   if constexpr (kWide) warpgroup_reg_dec<kIssueRegs>();
   if (warp == kEpiWarps) {
    // ------------------------------------------------------------ TMA producer (one thread per CTA)
    if (lane == 0) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_w);
      if constexpr (kSplit) {
        tma_prefetch_desc(&low.a);
        tma_prefetch_desc(&low.w);
      }
      auto load_w = [&](uint8_t* dst, int kc, const SplitWalk& w, uint64_t* bar, int n0) {
        if constexpr (kSplit) tma_load_2d_pair(dst, w.w_low() ? &low.w : &tmap_w, bar, w.k * kBlockK, n0);
        else tma_load_2d_pair(dst, &tmap_w, bar, kc * kBlockK, n0);
      };
      int stage = 0;
      uint32_t phase = 0;
      // The W slices of the first stages do not depend on the kernel in front: they are requested before the wait.
      const int ahead = u_count > 0 ? (k_chunks < kStages ? k_chunks : kStages) : 0;
      SplitWalk first(part_chunks, 0);
      for (int kc = 0; kc < ahead; ++kc, first.next()) {
        if (leader) mbar_arrive_expect_tx(&bars->full[kc], 2 * kStageBytes);
        load_w(smem_stage + kc * kStageBytes + kABytes, kc, first, &bars->full[kc], (pair % n_tiles) * kBlockN + static_cast<int>(rank) * kHalfN);
      }
      griddep_wait();
      for (int i = 0; i < u_count; ++i) {
        const int u = pair + i * n_pairs, row_tile = u / n_tiles, ntile = u % n_tiles;
        const int m0 = (2 * row_tile + static_cast<int>(rank)) * kBlockM;
        const int n0 = ntile * kBlockN + static_cast<int>(rank) * kHalfN;
        SplitWalk w(part_chunks, 0);
        for (int kc = 0; kc < k_chunks; ++kc, w.next()) {
          const bool early = i == 0 && kc < ahead;
          if (!early) {
            mbar_wait(&bars->empty[stage], phase ^ 1u, ctl, status, kErrWaitConsumer);
            if (leader) mbar_arrive_expect_tx(&bars->full[stage], 2 * kStageBytes);
          }
          uint8_t* dst = smem_stage + stage * kStageBytes;
          if constexpr (kSplit) {
            // a row of the product continues in the matrix's next row
            tma_load_2d_pair(dst, w.a_low() ? &low.a : &tmap_a, &bars->full[stage], w.k % args.rows.a_chunks * kBlockK, m0 + w.k / args.rows.a_chunks);
          } else {
            tma_load_2d_pair(dst, &tmap_a, &bars->full[stage], kc * kBlockK, m0);
          }
          if (!early) load_w(dst + kABytes, kc, w, &bars->full[stage], n0);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
   } else if (warp == kEpiWarps + 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    // The whole warp walks the loop and one elected lane issues (warp-uniform control flow keeps the descriptors in
    // uniform registers; a single lane under a lane test issues the same sequence a third slower).
    if (leader) {
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < u_count * n_acc; ++i) {            // accumulators, taken by the buffers in turn
        const int buf = i & 1;
        const uint32_t use = static_cast<uint32_t>(i >> 1);
        mbar_wait(&bars->acc_empty[buf], (use & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * kBlockN);
        for (int kc = 0; kc < acc_chunks; ++kc) {
          mbar_wait(&bars->full[stage], phase, ctl, status, kErrWaitTma);
          tc_fence_after_sync();
          const uint32_t base = smem_u32(smem_stage + stage * kStageBytes);
          const uint64_t a_desc = umma_desc_sw128(base);
          const uint64_t b_desc = umma_desc_sw128(base + kABytes);
#pragma unroll
          for (int ks = 0; ks < kBlockK / 16; ++ks) {
            if (elected) tc_mma_ss_pair(d_tmem, a_desc + 2u * ks, b_desc + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
          }
          if (elected) tc_commit_pair(&bars->empty[stage], 3);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (elected) tc_commit_pair(&bars->acc_full[buf], 3);
      }
    }
   }
  } else {
    // ------------------------------------------------------------ epilogue (warps 0..15 of both CTAs)
    if constexpr (kWide) warpgroup_reg_inc<kEpiRegs>();
    const int lg = warp & 3;      // TMEM lane group: rows 32*lg .. 32*lg+31 of the tile
    const int gsel = warp >> 2;   // which of the unit's four 64-column groups (wide), or which two (narrow)
    const uint32_t acc_empty_leader = map_to_cta(smem_u32(&bars->acc_empty[0]), 0);
    uint8_t* slab = smem_out + warp * kSlabBytes;
    bool done = false;
    if constexpr (kOut != 3) {
      if (kSplit || args.resid != nullptr) {
        // With a residual, accumulator rows cross the slab so that every lane finishes four columns of eight rows, and
        // residual and result are read and written as whole 128-byte (16 bit: 64-byte) lines by neighbouring lanes.  When
        // each lane fetched its own row's residual a load instruction touched 32 cache lines: 17 us of load-unit time per
        // 256 x 256 unit, more than its products take at K = 2048 (o_proj with an FP32 stream: 14 us at any row count).
        // A piece's residual (32 columns) is asked for one piece ahead.
        done = true;
        using T16 = typename std::conditional<kOut == 1, __half, __nv_bfloat16>::type;
        using R = typename std::conditional<kF32, float4, uint2>::type;             // four values
        constexpr int kElem = kF32 ? 4 : 2, kPieces = 2 * kGroupsPerWarp;
        const int r0 = lg * 32 + (lane >> 3), c4 = 4 * (lane & 7);
        const int n_pieces = u_count * kPieces;
        auto first_row = [&](int i) { return (2 * ((pair + i * n_pairs) / n_tiles) + static_cast<int>(rank)) * kBlockM + r0; };
        auto first_col = [&](int i, int p) { return ((pair + i * n_pairs) % n_tiles) * kBlockN + (gsel * kPieces + p) * 32 + c4; };
        auto fetch = [&](int idx, R (&r)[8]) {
          if (kSplit) return;
          const int i = idx / kPieces, row = first_row(i);
          const uint8_t* src = static_cast<const uint8_t*>(args.resid) + (static_cast<long long>(row) * args.N + first_col(i, idx % kPieces)) * kElem;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (row + 4 * k < args.M) r[k] = __ldcg(reinterpret_cast<const R*>(src + static_cast<long long>(4 * k) * args.N * kElem));
        };
        R res[8];
        if (n_pieces > 0) fetch(0, res);
#pragma unroll 1
        for (int idx = 0; idx < n_pieces; ++idx) {
          const int i = idx / kPieces, p = idx % kPieces, buf = n_acc == 2 ? 0 : i & 1;
          if (p == 0) {
            const uint32_t parity = static_cast<uint32_t>(n_acc == 2 ? i : i >> 1) & 1u;
            mbar_wait(&bars->acc_full[buf], parity, ctl, status, kErrWaitMma);
            if (n_acc == 2) mbar_wait(&bars->acc_full[1], parity, ctl, status, kErrWaitMma);
            tc_fence_after_sync();
          }
          uint32_t acc[32];
          const uint32_t t_piece = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + static_cast<uint32_t>(buf * kBlockN + (gsel * kPieces + p) * 32);
          tmem_ld32(t_piece, acc);
          R next[8];
          if (idx + 1 < n_pieces) fetch(idx + 1, next);
          const int col = first_col(i, p);
          const bool scaled = !kSplit && args.scale.data != nullptr;
          uint4 sc_raw = make_uint4(0u, 0u, 0u, 0u);
          if (scaled) sc_raw = args.scale.raw4<kF32>(col);
          tmem_ld_wait();
          if constexpr (kSplit) {
            if (n_acc == 2) {
              uint32_t other[32];
              tmem_ld32(t_piece + kBlockN, other);
              tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; ++c) acc[c] = __float_as_uint(__uint_as_float(acc[c]) + __uint_as_float(other[c]));
            }
          }
          if (p == kPieces - 1) {
            // Last read of the accumulator by this warp: hand it back before the arithmetic and the stores.
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive_cluster_relaxed(acc_empty_leader + static_cast<uint32_t>(buf) * 8u);
              if (n_acc == 2) mbar_arrive_cluster_relaxed(acc_empty_leader + 8u);
            }
          }
          float v[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = __uint_as_float(acc[c]);
          if constexpr (kSplit) {
            if (args.rows.by_channel) {           // neighbouring lanes hold neighbouring frames of a channel
              const int chan0 = ((pair + i * n_pairs) % n_tiles) * kBlockN + (gsel * kPieces + p) * 32;
              const long long at = args.rows.out_at((2 * ((pair + i * n_pairs) / n_tiles) + static_cast<int>(rank)) * kBlockM + lg * 32 + lane,
                                                    args.M, args.N);
              float* dst = static_cast<float*>(args.y) + at + static_cast<long long>(chan0) * args.rows.clip_valid;
              if (at >= 0) {
#pragma unroll
                for (int c = 0; c < 32; ++c) dst[static_cast<long long>(c) * args.rows.clip_valid] = v[c];
              }
              continue;
            }
          }
          if (!kSplit && args.gelu) {
#pragma unroll
            for (int c = 0; c < 32; c += 2) gelu_erf2(v[c], v[c + 1]);
          }
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<float4*>(slab + sw128_offset(lane, c)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
          __syncwarp();
          const float4 sc = scaled ? args.scale.value4<kF32>(sc_raw) : make_float4(1.f, 1.f, 1.f, 1.f);
          const int row = first_row(i);
          uint8_t* dst = static_cast<uint8_t*>(args.y) + (static_cast<long long>(row) * args.N + col) * kElem;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float4 o = *reinterpret_cast<const float4*>(slab + sw128_offset(4 * k + (lane >> 3), lane & 7));
            if constexpr (kSplit) {
              const int at = args.rows.out_row(row + 4 * k, args.M);
              if (at >= 0) *reinterpret_cast<float4*>(static_cast<float*>(args.y) + args.rows.at(at, col)) = o;
              continue;
            }
            o.x *= sc.x; o.y *= sc.y; o.z *= sc.z; o.w *= sc.w;
            if constexpr (kF32) {
              o.x += res[k].x; o.y += res[k].y; o.z += res[k].z; o.w += res[k].w;
              if (row + 4 * k < args.M) *reinterpret_cast<float4*>(dst + static_cast<long long>(4 * k) * args.N * 4) = o;
            } else {
              const float2 ra = Pack16<T16>::unpack(res[k].x), rb = Pack16<T16>::unpack(res[k].y);
              if (row + 4 * k < args.M)
                *reinterpret_cast<uint2*>(dst + static_cast<long long>(4 * k) * args.N * 2) =
                    make_uint2(Pack16<T16>::pack(o.x + ra.x, o.y + ra.y), Pack16<T16>::pack(o.z + rb.x, o.w + rb.y));
            }
            res[k] = next[k];
          }
          __syncwarp();
        }
      }
    }
    for (int i = 0; !done && i < u_count; ++i) {
      const int u = pair + i * n_pairs, row_tile = u / n_tiles, ntile = u % n_tiles;
      const int m0 = (2 * row_tile + static_cast<int>(rank)) * kBlockM;
      const long long row = static_cast<long long>(m0) + lg * 32 + lane;
      const bool row_ok = row < args.M;
      const int buf = i & 1;
      const uint32_t use = static_cast<uint32_t>(i >> 1);
      mbar_wait(&bars->acc_full[buf], use & 1u, ctl, status, kErrWaitMma);
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + static_cast<uint32_t>(buf * kBlockN);
#pragma unroll 1
      for (int g = gsel * kGroupsPerWarp; g < (gsel + 1) * kGroupsPerWarp; ++g) {
        const int col0 = ntile * kBlockN + g * 64;         // first output channel of this group
        uint32_t raw_lo[32], raw_hi[32];
        tmem_ld32(t_row + g * 64, raw_lo);
        tmem_ld32(t_row + g * 64 + 32, raw_hi);
        tmem_ld_wait();
        if (g == (gsel + 1) * kGroupsPerWarp - 1) {
          // Last read of the accumulator by this warp: hand it back before the arithmetic and the stores.
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty_leader + static_cast<uint32_t>(buf) * 8u);
        }
        float v[64];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          v[c] = __uint_as_float(raw_lo[c]);
          v[32 + c] = __uint_as_float(raw_hi[c]);
        }
        if constexpr (kOut == 3) {
          // approximate distances of this row to entries col0 .. col0 + 63, their minimum and who is within the margin
          const float4* q4 = reinterpret_cast<const float4*>(static_cast<const float*>(args.scale.data) + col0);        // same address in every lane
          float dmin = INFINITY;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float4 q = __ldg(q4 + j);
            v[4 * j] = fmaf(-2.f, v[4 * j], q.x); v[4 * j + 1] = fmaf(-2.f, v[4 * j + 1], q.y);
            v[4 * j + 2] = fmaf(-2.f, v[4 * j + 2], q.z); v[4 * j + 3] = fmaf(-2.f, v[4 * j + 3], q.w);
            dmin = fminf(dmin, fminf(fminf(v[4 * j], v[4 * j + 1]), fminf(v[4 * j + 2], v[4 * j + 3])));
          }
          const float limit = dmin + (row_ok ? __ldcg(static_cast<const float*>(args.resid) + row) : 0.f);
          uint32_t m_lo = 0u, m_hi = 0u;
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            m_lo |= (v[c] <= limit ? 1u : 0u) << c;
            m_hi |= (v[32 + c] <= limit ? 1u : 0u) << c;
          }
          if (row_ok)
            args.records[row * (args.N / 64) + (col0 >> 6)] = make_uint4(__float_as_uint(dmin), m_lo, m_hi, 0u);
          continue;
        }
        if (args.gelu) {
#pragma unroll
          for (int c = 0; c < 64; c += 2) gelu_erf2(v[c], v[c + 1]);
        }
        if (args.scale.data != nullptr) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float4 s = args.scale.load4(col0 + 4 * j);         // same address in every lane
            v[4 * j] *= s.x; v[4 * j + 1] *= s.y; v[4 * j + 2] *= s.z; v[4 * j + 3] *= s.w;
          }
        }
        if constexpr (kF32) {
          // FP32 output: two 32-column halves (128-byte rows) through the same 4 KB slab.
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (lane == 0) bulk_wait_group_read<0>();
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              *reinterpret_cast<float4*>(slab + sw128_offset(lane, c)) =
                  make_float4(v[h * 32 + 4 * c], v[h * 32 + 4 * c + 1], v[h * 32 + 4 * c + 2], v[h * 32 + 4 * c + 3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&tmap_y, slab, col0 + h * 32, m0 + lg * 32);   // rows past M are clipped
              bulk_commit_group();
            }
          }
        } else {
          using T16 = typename std::conditional<kOut == 1, __half, __nv_bfloat16>::type;
          if (lane == 0) bulk_wait_group_read<0>();
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            *reinterpret_cast<uint4*>(slab + sw128_offset(lane, c)) =
                make_uint4(Pack16<T16>::pack(v[8 * c], v[8 * c + 1]), Pack16<T16>::pack(v[8 * c + 2], v[8 * c + 3]),
                           Pack16<T16>::pack(v[8 * c + 4], v[8 * c + 5]), Pack16<T16>::pack(v[8 * c + 6], v[8 * c + 7]));
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmap_y, slab, col0, m0 + lg * 32);
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

static int encode_2d(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, uint64_t rows,
                     uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * static_cast<uint64_t>(elem_bytes)};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return encode_tiled(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int kOut, bool kWide, int kBlockN>
static int launch_pairs(const void* a, const void* w, const SplitLow* low, void* y, const LinearArgs& args, int pair_tiles, int max_pairs, int in_dtype,
                        int out_dtype, int* status, cudaStream_t st, int dependent) {
  using namespace lin;
  using S = Shape<kWide, kBlockN>;
  CUtensorMap tmap_a, tmap_w, tmap_y;
  SplitMaps<kOut == 4> low_maps = {};
  const CUtensorMapDataType t16 = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;   // any 16-bit element type moves alike
  const uint64_t M = static_cast<uint64_t>(args.M), N = static_cast<uint64_t>(args.N), K = static_cast<uint64_t>(args.K);
  const uint64_t a_rows = kOut == 4 ? static_cast<uint64_t>(low->a_rows) : M;
  const uint64_t a_cols = kOut == 4 ? static_cast<uint64_t>(args.rows.a_chunks) * kBlockK : K;
  int rc = encode_2d(&tmap_a, t16, 2, a, a_rows, a_cols, kBlockM, kBlockK);
  if (rc != 0) return rc;
  rc = encode_2d(&tmap_w, t16, 2, w, N, K, S::kHalfN, kBlockK);
  if (rc != 0) return rc;
  if constexpr (kOut == 4) {
    rc = encode_2d(&low_maps.a, t16, 2, low->a, a_rows, a_cols, kBlockM, kBlockK);
    if (rc == 0) rc = encode_2d(&low_maps.w, t16, 2, low->w, N, K, S::kHalfN, kBlockK);
    if (rc != 0) return rc;
  }
  if (out_dtype >= 3)      // no tiled store in these modes: a placeholder map over a
    rc = encode_2d(&tmap_y, t16, 2, a, a_rows, a_cols, 32, 64);
  else if (out_dtype == 2)
    rc = encode_2d(&tmap_y, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, y, M, N, 32, 32);
  else
    rc = encode_2d(&tmap_y, t16, 2, y, M, N, 32, 64);
  if (rc != 0) return rc;
  const int total_units = pair_tiles * (args.N / kBlockN);
  const int n_pairs = total_units < max_pairs ? total_units : max_pairs;
  const int fmt = in_dtype == 1 ? 0 : 1;   // tcgen05 kind::f16 operand format: 0 = F16, 1 = BF16
  const uint32_t idesc = umma_idesc_f16(2 * kBlockM, kBlockN, fmt, fmt, 0, 0);
  auto kern = linear_gemm_kernel<kOut, kWide, kBlockN>;
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), S::kSmemBytes);
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(2 * n_pairs), S::kThreads, S::kSmemBytes, st, 1, dependent, tmap_a, tmap_w, tmap_y, low_maps,
                       args, total_units, idesc, status);
}

// 256 x 128 units instead of 256 x 256 where they save part of a wave in a call whose rows cross the slab (a residual, a
// split-precision product): there a half unit costs about half plus 1 / 128 per K chunk of a whole one (its a slices are fetched
// twice as often).  Without the slab it costs two thirds to three quarters, and no wave that it saves is worth that.  (One wave
// of them: see one_wave_of_halves.)  Measured, whole -> half units, in us:
//   residual         K =  512, N =  512, 12000 rows (2 -> 3 waves) 18.8 -> 16.7, 22000 rows (3 -> 5) 31.8 -> 29.1
//                    K = 1024, N = 1024, FP16, 5000 rows (2 -> 3) 27.2 -> 24.2, 16000 rows (4 -> 7) 38.7 -> 42.9
//                    K = 2048, N =  512, 14000 rows (2 -> 3) 35.2 -> 36.7, 22000 rows (3 -> 5) 49.9 -> 56.2
//   split precision  K =  256, N =  512, 12000 rows (2 -> 3) 29.3 -> 25.0;  K = 512, 33.2 -> 37.1;  K = 2048, 84.4 -> 113.1
//   neither          K =  512, N =  512, 12000 rows (2 -> 3) 12.6 -> 14.6;  K = 1024, N = 1024, 16000 rows (4 -> 7) 29.0 -> 37.2
static bool half_units(int pair_tiles, int N, int max_pairs, int k_chunks) {
  const int waves256 = (pair_tiles * (N / 256) + max_pairs - 1) / max_pairs, waves128 = (pair_tiles * (N / 128) + max_pairs - 1) / max_pairs;
  return static_cast<long long>(64 + k_chunks) * waves128 < 128ll * waves256;
}

// (What fm_linear_ws.cu takes comes first; the figures are for the other kernels alone.)
// Half units that are one wave, for rows that two of the few-row kernel's 128 x 64 blocks on an SM would hold: those fetch half as much
// again from L2, and the second starts when the first has gone.  With one of them to an SM they are the faster form.  Measured, few-row
// kernel -> half units, in us: K = 2048, N = 512, FP32 2000 rows (128 blocks) 12.4 -> 13.9, 2500 (160) 13.9 -> 13.9, 3678 (232) 15.7 ->
// 14.0, 4500 (288) 16.7 -> 14.2, BF16 3678 rows 16.7 -> 14.4; K = 512, N = 512, FP32 3678 rows 8.8 -> 8.3, BF16 9.8 -> 8.5; K = 512,
// N = 2048, GELU 500 rows (128) 8.0 -> 8.3, 1024 (256) 9.8 -> 8.3.
// FP32 results of rows that hardly give any SM a second block are out sooner from the few-row kernel, whose last blocks are short where
// their rows are few, in a call by itself: K = 2048, N = 512 2305 rows 12.9 -> 14.0, 2400 13.1 -> 13.9, K = 512, N = 512 2400 rows 7.5 -> 8.1, N = 1024
// 1153 rows 7.3 -> 7.8, 1280 8.0 -> 7.8, N = 2048 513 rows 7.3 -> 7.8.  16-bit ones are not (K = 2048, N = 512 2400 rows 14.0 -> 14.0, K = 512 8.6 ->
// 8.4, N = 2048, GELU 513 rows 8.3 -> 8.1), nor in a chain, whose next kernel finds an SM free the sooner (8 layers of 2313 rows 452 -> 430).  What
// a chain leaves to this rule of products with GELU is beyond the rows that have resident weights (8 layers, few-row kernel -> half units, FP32 and
// BF16 streams: MLP of 2048 769 rows 315 -> 308 and 319 -> 311, 1000 331 -> 325 and 331 -> 325; of 1024 1537 rows 383 -> 373 and 393 -> 384; of 1280 1153 rows 345 -> 345 and 359 -> 355; of 2304
// 641 307 -> 303 and 315 -> 311; of 2560 513 295 -> 291 and 304 -> 297; of 3328 385 278 -> 281 and 283 -> 283, 466 285 -> 278 and 286 -> 282; of 3840 385 286 -> 289 and 291 -> 292).
static bool one_wave_of_halves(int M, int pair_tiles, int N, int max_pairs, bool fp32, int dependent) {
  constexpr int kBlock = lin::kBlockM * 64;
  const long long sms = sm_count(), results = static_cast<long long>(M) * N;
  if (pair_tiles * static_cast<long long>(N / 128) > max_pairs) return false;
  if (fp32 && !dependent) return results > kBlock * 33 / 32 * sms;
  return static_cast<long long>((M + lin::kBlockM - 1) / lin::kBlockM) * (N / 64) > sms;
}

int launch_linear_gemm(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N,
                       int K, int in_dtype, int out_dtype, int gelu, int* status, cudaStream_t st, int dependent) {
  using namespace lin;
  if (M < 0 || N <= 0 || K <= 0 || N % 256 != 0 || K % kBlockK != 0) return -1;
  if (in_dtype < 0 || in_dtype > 1 || out_dtype < 0 || out_dtype > 3) return -1;
  if (M == 0) return 0;
  if (a == nullptr || w == nullptr || y == nullptr) return -1;
  if (out_dtype == 3 && (scale.data == nullptr || scale.type != 2 || resid == nullptr || gelu)) return -1;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) |
       reinterpret_cast<uintptr_t>(scale.data) | reinterpret_cast<uintptr_t>(resid)) & 15u)
    return -3;
  if (out_dtype != 3 && linear_ws_takes(M, N, K, dependent, resid != nullptr && out_dtype != 2))
    return launch_linear_ws(a, w, y, scale, resid, M, N, K, in_dtype, out_dtype, gelu, status, st, dependent);
  const int pair_tiles = ((M + kBlockM - 1) / kBlockM + 1) / 2;
  const int max_pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  const bool one_wave = out_dtype != 3 && one_wave_of_halves(M, pair_tiles, N, max_pairs, out_dtype == 2, dependent);
  if (out_dtype != 3 && !one_wave && few_row_tiles(M, N))
    return launch_linear_small(a, w, y, scale, resid, M, N, K, in_dtype, out_dtype, gelu, status, st, dependent);
  // The wide shape where the epilogue carries arithmetic (GELU, candidate records) for unit after unit, the narrow one otherwise.
  const bool wide = !one_wave && (gelu || out_dtype == 3);
  const bool halves = one_wave || (!wide && resid != nullptr && half_units(pair_tiles, N, max_pairs, K / kBlockK));
  LinearArgs args = {scale, resid, M, N, K, gelu ? 1 : 0, out_dtype == 3 ? static_cast<uint4*>(y) : nullptr, y, {}};
  using Fn = int (*)(const void*, const void*, const SplitLow*, void*, const LinearArgs&, int, int, int, int, int*, cudaStream_t, int);
  Fn fn;
  if (wide)
    fn = out_dtype == 3 ? launch_pairs<3, true, 256>
                        : (out_dtype == 2 ? launch_pairs<2, true, 256> : (out_dtype == 1 ? launch_pairs<1, true, 256> : launch_pairs<0, true, 256>));
  else if (halves)
    fn = out_dtype == 2 ? launch_pairs<2, false, 128> : (out_dtype == 1 ? launch_pairs<1, false, 128> : launch_pairs<0, false, 128>);
  else
    fn = out_dtype == 2 ? launch_pairs<2, false, 256> : (out_dtype == 1 ? launch_pairs<1, false, 256> : launch_pairs<0, false, 256>);
  return fn(a, w, nullptr, y, args, pair_tiles, max_pairs, in_dtype, out_dtype, status, st, dependent);
}

int launch_linear_split(const void* a_hi, const void* a_lo, long long a_rows, int a_cols, const void* w_hi, const void* w_lo, float* y,
                        long long rows, int clip_rows, int clip_valid, int by_channel, int n_mats, int parts, int N, int K, int* status,
                        cudaStream_t st, int dependent) {
  using namespace lin;
  if (rows < 0 || a_rows > 0x7fffffffLL || a_rows < rows || N <= 0 || K <= 0 || N % 256 != 0 || a_cols <= 0 || a_cols % kBlockK != 0 ||
      K % a_cols != 0 || n_mats <= 0 || N % (256 * n_mats) != 0 || (by_channel && n_mats != 1) || parts < 1 || parts > 2 ||
      K % (parts * kBlockK) != 0 || clip_rows <= 0 || clip_valid <= 0 || clip_valid > clip_rows)
    return -1;
  if (rows == 0) return 0;
  if (a_hi == nullptr || a_lo == nullptr || w_hi == nullptr || w_lo == nullptr || y == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(a_hi) | reinterpret_cast<uintptr_t>(a_lo) | reinterpret_cast<uintptr_t>(w_hi) |
       reinterpret_cast<uintptr_t>(w_lo) | reinterpret_cast<uintptr_t>(y)) & 15u)
    return -3;
  const int M = static_cast<int>(rows);
  const SplitLow low = {a_lo, w_lo, a_rows};
  const long long results = (rows + clip_rows - 1) / clip_rows * clip_valid - (rows % clip_rows != 0 && rows % clip_rows < clip_valid ? clip_valid - rows % clip_rows : 0);
  const SplitRows map = {a_cols / kBlockK, clip_rows, clip_valid, by_channel, parts, N / n_mats, results * (N / n_mats)};
  if (few_row_tiles(M, N)) return launch_linear_split_small(a_hi, w_hi, low, map, y, M, N, K, status, st, dependent);
  const int pair_tiles = ((M + kBlockM - 1) / kBlockM + 1) / 2;
  const int max_pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  const LinearArgs args = {ParamVec(nullptr), nullptr, M, N, K, 0, nullptr, y, map};
  auto fn = half_units(pair_tiles, N, max_pairs, 3 * (K / kBlockK)) ? launch_pairs<4, false, 128> : launch_pairs<4, false, 256>;
  return fn(a_hi, w_hi, &low, y, args, pair_tiles, max_pairs, 1, 4, status, st, dependent);
}

}  // namespace fm
