// Split-precision products that make their operand on the way (sm_100a): y = A W^T in FP32 grade from FP16 tensor-core products, where
// A is FP32 rows, or the frames that a strided convolution sees.
//
// As kernels of their own (fm_downsample.cu, fm_rvq.cu, then fm_linear_gemm.cu) the FP16 hi and lo parts of A went through memory: for
// 64000 rows 88 us of 385 in front of a convolution (K = 2048, N = 512; here 302 in all, 1.33 PFLOP/s over the three terms, which is what
// the power limit leaves), 41 of 137 in front of a projection (K = 512; here 112, where the epilogue's loads hold up every eighth slice).  And with one accumulator K has to run three
// times, so that the small terms are summed first: hi of A and of W crossed L2 twice.  Here sixteen warps read A as it lies, split it
// into the two operand tiles in shared memory, and a slice of 64 dimensions is multiplied once: lo W_hi and hi W_lo into one accumulator,
// hi W_hi into another, added in FP32 at the end.  That is 64 KB a slice and block out of L2 instead of 96, and no more error: each
// accumulator takes fewer sums.
//
// A pair of blocks (cta_group::2) owns 256 rows x 256 outputs, 512 columns of tensor memory, so the next unit's products wait for the
// epilogue's loads: by then three slices of it are in place, and the stores follow beside its products.
//
// Warps 0-15: operand A, epilogue.  Warp 16: W.  Warp 17: MMA (leader block only).
#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"

namespace fm {

namespace sg {
constexpr int kBlockM = 128, kBlockN = 256, kBlockK = 64;
constexpr int kWorkers = 16, kThreads = (kWorkers + 4) * 32;
constexpr int kWorkRegs = 112, kIssueRegs = 32;
static_assert(512 * kWorkRegs + 128 * kIssueRegs <= kThreads * 96, "register pool of the launch");
constexpr int kTileBytes = kBlockM * kBlockK * 2;              // of A, or of this block's half of W
constexpr int kStages = 3, kStageBytes = 4 * kTileBytes;       // A hi, A lo, W hi, W lo
constexpr int kTmemCols = 512;                                 // the small terms' accumulator, then hi W_hi's
struct Barriers {
  uint64_t w_full[kStages], peer_full[kStages];                // in the leader: W of both blocks, A of the other one
  uint64_t a_full[kStages], empty[kStages];                    // per block
  uint64_t acc_full, acc_empty;                                // acc_empty: in the leader
  uint32_t tmem_base, skip;
  CtaCtl ctl;
  int2 place[2][2][kBlockM];                                   // per group and of two units: a row's clip and its first frame
};
constexpr int kSmemBytes = 1024 + kStages * kStageBytes + static_cast<int>(sizeof(Barriers));
}  // namespace sg

struct SplitSource {
  const float* x;              // rows [M, K]; or frames [.., T, C]
  int T, T_out, C, stride, left;         // frames: row t of a clip sees frames t * stride - left .., clamped to the clip
};
struct SplitGemmArgs {
  SplitSource src;
  float* y;
  int M, N, K;
  int cols;                    // of one of the matrices that the outputs make
  long long mat_step;
};

// kSource: 0 = rows, 1 = frames of a convolution
template <int kSource>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sg::kThreads, 1)
split_gemm_kernel(const __grid_constant__ CUtensorMap tmap_hi, const __grid_constant__ CUtensorMap tmap_lo,
                  const __grid_constant__ SplitGemmArgs args, int total_units, uint32_t idesc, int* status) {
  using namespace sg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + kStages * kStageBytes);
  CtaCtl* ctl = &bars->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = rank == 0;
  const int n_tiles = args.N / kBlockN, k_chunks = args.K / kBlockK;
  // round-robin: neighbouring pairs work on the output tiles of the same rows, which come from memory once
  const int pair = static_cast<int>(blockIdx.x >> 1), n_pairs = static_cast<int>(gridDim.x >> 1);
  const int u_count = (total_units - pair + n_pairs - 1) / n_pairs;
  auto unit = [&](int i) { return pair + i * n_pairs; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->w_full[i], 1);
      mbar_init(&bars->peer_full[i], 1);
      mbar_init(&bars->a_full[i], kWorkers / 2);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->acc_empty, 2 * kWorkers);
    ctl->abort = 0;
    bars->skip = (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0) ? 1u : 0u;
    fence_mbar_init();
  }
  if (warp == kWorkers) {
    tmem_alloc_pair(&bars->tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  const bool skip = ld_shared_cluster_u32(map_to_cta(smem_u32(&bars->skip), 0)) != 0;

  if (skip) {
    // a kernel in front already reported an error through this status word: do nothing
  } else if (warp >= kWorkers) {
    warpgroup_reg_dec<kIssueRegs>();
    if (warp == kWorkers && lane == 0) {
      // ---------------------------------------------------------- W
      tma_prefetch_desc(&tmap_hi);
      tma_prefetch_desc(&tmap_lo);
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < u_count; ++i) {
        const int n0 = unit(i) % n_tiles * kBlockN + static_cast<int>(rank) * (kBlockN / 2);
#pragma unroll 1
        for (int kc = 0; kc < k_chunks; ++kc) {
          mbar_wait(&bars->empty[stage], phase ^ 1u, ctl, status, kErrWaitConsumer);
          if (leader) mbar_arrive_expect_tx(&bars->w_full[stage], 4 * kTileBytes);
          uint8_t* dst = smem + stage * kStageBytes + 2 * kTileBytes;
          tma_load_2d_pair(dst, &tmap_hi, &bars->w_full[stage], kc * kBlockK, n0);
          tma_load_2d_pair(dst + kTileBytes, &tmap_lo, &bars->w_full[stage], kc * kBlockK, n0);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    } else if (warp == kWorkers + 1 && leader) {
      // ---------------------------------------------------------- products
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < u_count; ++i) {
        mbar_wait(&bars->acc_empty, (static_cast<uint32_t>(i) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
        tc_fence_after_sync();
#pragma unroll 1
        for (int kc = 0; kc < k_chunks; ++kc) {
          mbar_wait(&bars->w_full[stage], phase, ctl, status, kErrWaitTma);
          mbar_wait(&bars->a_full[stage], phase, ctl, status, kErrWaitConsumer);
          mbar_wait_cluster(&bars->peer_full[stage], phase, ctl, status, kErrWaitConsumer);
          tc_fence_after_sync();
          const uint32_t base = smem_u32(smem + stage * kStageBytes);
          const uint64_t a_hi = umma_desc_sw128(base), a_lo = umma_desc_sw128(base + kTileBytes);
          const uint64_t w_hi = umma_desc_sw128(base + 2 * kTileBytes), w_lo = umma_desc_sw128(base + 3 * kTileBytes);
#pragma unroll
          for (int ks = 0; ks < kBlockK / 16; ++ks) {
            if (elected) {
              tc_mma_ss_pair(tmem_base, a_lo + 2u * ks, w_hi + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
              tc_mma_ss_pair(tmem_base, a_hi + 2u * ks, w_lo + 2u * ks, idesc, 1u);
              tc_mma_ss_pair(tmem_base + kBlockN, a_hi + 2u * ks, w_hi + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
            }
          }
          if (elected) tc_commit_pair(&bars->empty[stage], 3);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (elected) tc_commit_pair(&bars->acc_full, 3);
      }
    } else if (warp == kWorkers + 1 && lane == 0) {
      // ---------------------------------------------------------- the other block's A: one arrival for its sixteen warps
      // (An arrival in another block's memory that releases is a fence over all that its thread has under way: 2000 cycles for a warp
      // with loads and stores in flight.)
      const uint32_t peer_full_leader = map_to_cta(smem_u32(&bars->peer_full[0]), 0);
      int stage = 0;
      uint32_t phase = 0;
#pragma unroll 1
      for (int c = 0; c < u_count * k_chunks; ++c) {
        mbar_wait(&bars->a_full[stage], phase, ctl, status, kErrWaitConsumer);
        mbar_arrive_cluster(peer_full_leader + static_cast<uint32_t>(stage) * 8u);
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------ operand A; epilogue
    // Two groups of eight warps take the slices in turn.  What a group loads for its next slice must not be under way when it hands
    // one over (the fence waits for it: 64000 rows, K = 2048, N = 512, all warps on every slice and loads two slices ahead 375 us, one ahead 305,
    // like this 302), so the other group's work hides it.
    warpgroup_reg_inc<kWorkRegs>();
    const SplitSource& src = args.src;
    const uint32_t acc_empty_leader = map_to_cta(smem_u32(&bars->acc_empty), 0);
    const int group = warp >> 3, r0 = (warp & 7) * 16 + (lane >> 4), piece = lane & 15;         // rows r0, r0 + 2 .., four dimensions of a slice
    auto tile_row = [&](int i) { return (2 * (unit(i) / n_tiles) + static_cast<int>(rank)) * kBlockM; };
    auto open_unit = [&](int i) {
      if constexpr (kSource == 1) {
        const int t = static_cast<int>(threadIdx.x) & 255;
        if (t < kBlockM) {
          const int row = tile_row(i) + t < args.M ? tile_row(i) + t : args.M - 1;
          const int clip = row / src.T_out;
          bars->place[group][i & 1][t] = make_int2(clip * src.T, (row - clip * src.T_out) * src.stride - src.left);
        }
        asm volatile("bar.sync %0, 256;" ::"r"(group + 1) : "memory");
      }
    };
    // Rows past the end repeat the last one (nobody reads what comes of them): a test here would make the loads wait for one another.
    auto fetch = [&](int i, int kc, float4 (&v)[8]) {
      if constexpr (kSource == 0) {
        const int m0 = tile_row(i) + r0;
        const float* p = src.x + kc * kBlockK + 4 * piece;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int row = m0 + 2 * k < args.M ? m0 + 2 * k : args.M - 1;
          v[k] = __ldg(reinterpret_cast<const float4*>(p + static_cast<long long>(row) * args.K));
        }
      } else {
        const int per_frame = src.C / kBlockK, j = kc / per_frame;
        const float* p = src.x + (kc - j * per_frame) * kBlockK + 4 * piece;
        int2 at[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) at[k] = bars->place[group][i & 1][r0 + 2 * k];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int f = max(0, min(at[k].y + j, src.T - 1));
          v[k] = __ldg(reinterpret_cast<const float4*>(p + static_cast<long long>(at[k].x + f) * src.C));
        }
      }
    };
    const int lg = warp & 3, g = warp >> 2;          // the epilogue's rows and 64 of its columns
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lg * 32) << 16) + static_cast<uint32_t>(g * 64);
    auto finish = [&](int i) {
      mbar_wait(&bars->acc_full, static_cast<uint32_t>(i) & 1u, ctl, status, kErrWaitMma);
      tc_fence_after_sync();
      uint32_t v[2][32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tmem_ld32(t_row + kBlockN + h * 32, v[h]);
        uint32_t low[16];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          tmem_ld16(t_row + h * 32 + part * 16, low);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) v[h][part * 16 + c] = __float_as_uint(__uint_as_float(low[c]) + __uint_as_float(v[h][part * 16 + c]));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty_leader);
      const int row = tile_row(i) + lg * 32 + lane, col = unit(i) % n_tiles * kBlockN + g * 64;
      if (row < args.M) {
        const int mat = col / args.cols;
        float* dst = args.y + mat * args.mat_step + static_cast<long long>(row) * args.cols + (col - mat * args.cols);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 4; ++c) st_global_v8(dst + h * 32 + 8 * c, v[h] + 8 * c);
      }
    };

    float4 v[8];
    if (u_count > 0) {
      open_unit(0);
      fetch(0, group, v);
    }
    for (int i = 0; i < u_count; ++i) {
#pragma unroll 1
      for (int kc = group; kc < k_chunks; kc += 2) {
        const int slice = i * k_chunks + kc, stage = slice % kStages;
        uint8_t* dst = smem + stage * kStageBytes + (piece & 1) * 8;
        mbar_wait(&bars->empty[stage], (static_cast<uint32_t>(slice / kStages) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t h0 = Pack16<__half>::pack(v[k].x, v[k].y), h1 = Pack16<__half>::pack(v[k].z, v[k].w);
          const float2 b0 = Pack16<__half>::unpack(h0), b1 = Pack16<__half>::unpack(h1);
          const uint32_t at = sw128_offset(static_cast<uint32_t>(r0 + 2 * k), static_cast<uint32_t>(piece >> 1));
          *reinterpret_cast<uint2*>(dst + at) = make_uint2(h0, h1);
          *reinterpret_cast<uint2*>(dst + kTileBytes + at) =
              make_uint2(Pack16<__half>::pack(v[k].x - b0.x, v[k].y - b0.y), Pack16<__half>::pack(v[k].z - b1.x, v[k].w - b1.y));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->a_full[stage]);
        if (i > 0 && kc == (group == 0 ? 2 : 1)) finish(i - 1);          // the stages hold the first three slices of this unit
        if (kc + 2 < k_chunks) {
          fetch(i, kc + 2, v);
        } else if (i + 1 < u_count) {
          open_unit(i + 1);
          fetch(i + 1, group, v);
        }
      }
    }
    if (u_count > 0) finish(u_count - 1);
  }

  // Neither block may leave (or release tensor memory) while its partner can still signal it.
  tc_fence_before_sync();
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);   // copies that may still be in flight get time to land
  cluster_sync_all();
  if (warp == kWorkers) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

template <int kSource>
static int launch_source(const SplitGemmArgs& args, const void* w_hi, const void* w_lo, int* status, cudaStream_t st) {
  using namespace sg;
  CUtensorMap hi, lo;
  int rc = encode_rows_16bit(&hi, w_hi, static_cast<uint64_t>(args.N), static_cast<uint64_t>(args.K), kBlockN / 2, kBlockK);
  if (rc == 0) rc = encode_rows_16bit(&lo, w_lo, static_cast<uint64_t>(args.N), static_cast<uint64_t>(args.K), kBlockN / 2, kBlockK);
  if (rc != 0) return rc;
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(split_gemm_kernel<kSource>), kSmemBytes);
  if (rc != 0) return rc;
  const int units = (args.M + 2 * kBlockM - 1) / (2 * kBlockM) * (args.N / kBlockN), pairs = sm_count() / 2 > 0 ? sm_count() / 2 : 1;
  return launch_kernel(split_gemm_kernel<kSource>, dim3(static_cast<unsigned>(2 * (units < pairs ? units : pairs))), kThreads, kSmemBytes, st, 1, 0, hi, lo,
                       args, units, umma_idesc_f16(2 * kBlockM, kBlockN, 0, 0, 0, 0), status);
}

// Whole tiles of 256 x 256, each a chain of K / 64 slices, against the tiles and splits of K that the other kernels have for few rows
// (K = 2048, N = 512: 1000 rows 37 us there, 49 here, 2500 rows 59 and 49; K = 512, N = 512: 2000 rows 25 and 25, 4800 rows 33 and 27;
// K = 512, N = 256: 4096 rows 27 and 27, 16000 rows 41 and 29).  With four slices the chain is little beside what a tile costs anyway,
// and the few-row tiles are faster as long as they are one wave (K = 256, in us on the GPU alone, there and here: N = 512, 2048 rows 13.6 and
// 15.7, 4736 rows 15.4 and 15.7, 5000 rows 20.1 and 15.8; N = 256, 4096 rows 13.6 and 15.7, 9472 rows 16.1 and 15.7, 12500 rows 22.0 and 16.2;
// K = 384, N = 256, 4096 rows 16.9 and 17.4, N = 1024, 2048 rows 17.9 and 17.9).  And for every 256 outputs A is split anew, which many outputs and few
// slices don't pay (K = 512, N = 4096: 2048 rows 35.3 and 33.6, 4096 rows 58.9 and 59.3, 8000 rows 92.8 and 98.0; N = 2048, 8000 rows 61.4 and
// 59.8, 24000 rows 146 and 148; K = 1024, N = 4096, 6000 rows 134 and 132).
bool split_gemm_takes(long long rows, int N, int K) {
  if (rows * N < 1ll << 20 || N % sg::kBlockN != 0 || K < 4 * sg::kBlockK || K % (2 * sg::kBlockK) != 0) return false;
  if (K == 4 * sg::kBlockK && rows <= 0x7fffffffLL && few_row_tiles(static_cast<int>(rows), N)) return false;
  return N < 2048 || K >= 1024 || rows * N <= 1ll << 24;
}

static bool bad_shape(long long rows, int N, int K) {
  return rows < 0 || rows > 0x7fffff00LL || N <= 0 || N % sg::kBlockN != 0 || K < 4 * sg::kBlockK || K % (2 * sg::kBlockK) != 0;
}
static bool misaligned(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) != 0 ||
         (reinterpret_cast<uintptr_t>(d) & 31u) != 0;
}

int launch_split_rows(const float* x, const void* w_hi, const void* w_lo, float* y, long long rows, int n_mats, int N, int K, int* status,
                      cudaStream_t st) {
  if (bad_shape(rows, N, K) || n_mats <= 0 || N % (sg::kBlockN * n_mats) != 0) return -1;
  if (rows == 0) return 0;
  if (x == nullptr || w_hi == nullptr || w_lo == nullptr || y == nullptr) return -1;
  if (misaligned(x, w_hi, w_lo, y)) return -3;
  SplitGemmArgs args = {};
  args.src.x = x;
  args.y = y;
  args.M = static_cast<int>(rows);
  args.N = N;
  args.K = K;
  args.cols = N / n_mats;
  args.mat_step = rows * args.cols;
  return launch_source<0>(args, w_hi, w_lo, status, st);
}

int launch_split_conv(const float* x, const void* w_hi, const void* w_lo, float* y, int B, int T, int C, int kernel, int stride, int N, int* status,
                      cudaStream_t st) {
  if (B < 0 || T < 0 || C <= 0 || C % sg::kBlockK != 0 || stride <= 0 || kernel < stride || kernel > 16) return -1;
  const int T_out = (T + stride - 1) / stride;
  const long long rows = static_cast<long long>(B) * T_out;
  if (bad_shape(rows, N, kernel * C)) return -1;
  if (rows == 0) return 0;
  if (x == nullptr || w_hi == nullptr || w_lo == nullptr || y == nullptr) return -1;
  if (misaligned(x, w_hi, w_lo, y)) return -3;
  SplitGemmArgs args = {};
  args.src.x = x;
  args.src.T = T;
  args.src.T_out = T_out;
  args.src.C = C;
  args.src.stride = stride;
  args.src.left = kernel - stride;
  args.y = y;
  args.M = static_cast<int>(rows);
  args.N = N;
  args.K = kernel * C;
  args.cols = N;
  return launch_source<1>(args, w_hi, w_lo, status, st);
}

}  // namespace fm
