// Linear layers and the QKV projection for few rows (sm_100a): y = residual + scale * act(a W^T), or q | k | v with
// RoPE, for calls whose rows fill only a few 128-row tiles (one clip, one frame of up to a few hundred streams).
//
// Where the weights fit the chip's tensor memory such calls take fm_linear_ws.cu.  Left to this kernel are split-precision products (the quantiser's
// projections and convolution), q | k | v of 769 rows and more (1025 in a layer's chain), K that is not 512 times a power of two, and linear
// layers past that kernel's lines: by themselves, FP32 with a residual, K = 2048, N = 512 600 rows 9.7 us, 1800 12.2.
//
// What bounds such a call is latency and the number of SMs that pull weights out of L2, not arithmetic: the pair
// kernels (fm_linear_gemm.cu, fm_qkv_gemm.cu) cut the output into 256 x 256 tiles, so that 125 rows x 512 outputs at
// K = 2048 occupied 4 of 148 SMs, each walking 32 K-chunks one after the other (with an FP32 residual 20.8 us; here 6.8 us, 6.0 with resident weights).  Here a block owns
// 128 rows x 64 outputs (one attention head; or x 32) and a SLICE of K: the blocks of a thread-block cluster share one output
// tile and split K between them, so the same layer runs on 64 SMs with four chunks each.  The partial sums meet in
// distributed shared memory: row r of the tile belongs to cluster rank r % S, every block sends its FP32 partials of an
// owner's rows with one bulk copy per warp and owner (single 16-byte remote stores took 1.5 us for a full tile), and the
// owner adds them in rank order (the result does not depend on timing), applies the epilogue and stores whole 64-byte
// segments.
//
// Weights do not depend on the kernel in front, so in a chain of dependent launches the W slices of the first stages
// are requested before the wait for that kernel and arrive while it still runs.  About 105 KB of shared memory and 64
// tensor-memory columns per block leave room for the next kernel's blocks on the same SM, which is what makes that
// overlap possible.
//
// Warps 0-3: accumulator rows out of tensor memory.  Warp 4: TMA.  Warp 5: MMA.  All six finish the owned rows.
#include "fm_launch.h"
#include "fm_small_tile.cuh"

namespace fm {

namespace small {
constexpr int kBlockM = 128;
constexpr int kBlockK = 64;
constexpr int kStages = 3;
constexpr int kABytes = kBlockM * kBlockK * 2;     // 16 KB
constexpr int kThreads = 192;
template <int kBlockN> struct Tile {
  static constexpr int kStageBytes = kABytes + kBlockN * kBlockK * 2;
  static constexpr int kRedBytes = kBlockM * kBlockN * 4;      // S sources x (128 / S) rows x FP32 columns
  static constexpr int kSmemBytes = 1024 + kStages * kStageBytes + kRedBytes + 128;
};

struct Barriers {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full;
  uint64_t red_full;         // the partial sums of this block's rows have arrived from every block of the cluster
  uint32_t tmem_base;
  CtaCtl ctl;
};
static_assert(sizeof(Barriers) <= 128, "barrier block too large");

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Copy from this block's shared memory into that of a block of the cluster (both addresses 16-byte aligned); the bytes are
// counted on a barrier of the destination.
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "r"(smem_u32(src)), "r"(bytes), "r"(bar) : "memory");
}
}  // namespace small

// kOut: 0 = BF16, 1 = FP16, 2 = FP32 output and residual; 3 = q | k | v with RoPE (VT: type of v); 4 = FP32 output of a
// split-precision product: K runs three times (lo W_hi, hi W_lo, hi W_hi; part by part), shared out like any other K
template <int kOut, typename VT, int kBlockN>
__global__ void __launch_bounds__(small::kThreads)
linear_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                    const __grid_constant__ SplitMaps<kOut == 4> low,
                    const __grid_constant__ SmallArgs args, uint32_t idesc, int* status) {
  using namespace small;
  constexpr int kStageBytes = Tile<kBlockN>::kStageBytes, kRedBytes = Tile<kBlockN>::kRedBytes, kTmemCols = (kOut == 4 ? 2 : 1) * kBlockN;
  constexpr int kHalves = kBlockN / 32;
  constexpr uint32_t kRowBytes = kBlockN * 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* red = smem + kStages * kStageBytes;
  Barriers* bars = reinterpret_cast<Barriers*>(red + kRedBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = args.split;
  const int rank = split > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int ntile = static_cast<int>(blockIdx.x) / split;
  const int n0 = ntile * kBlockN;
  const int m0 = static_cast<int>(blockIdx.y) * kBlockM;
  const int chunk0 = rank * args.chunks;
  // Two parts of a split-precision product in one block have an accumulator each; shared out over an even number of blocks,
  // every block has chunks of one part.
  const bool two_acc = kOut == 4 && args.rows.parts == 2 && split == 1;
  // Row r of the tile belongs to rank r % S.
  const int log_s = 31 - __clz(split);
  const int valid = args.M - m0 < kBlockM ? args.M - m0 : kBlockM;
  const int n_own = (valid - rank + split - 1) >> log_s;

  // read early: a status set before this chain began stops every kernel of it (the stores are left out)
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->red_full, 1);
    bars->ctl.abort = 0;
    fence_mbar_init();
    if (split > 1 && n_own > 0) mbar_arrive_expect_tx(&bars->red_full, static_cast<uint32_t>(split * n_own) * kRowBytes);
  }
  if (warp == 5) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (split > 1) cluster_arrive();        // "this block runs": its shared memory may be written from now on
  griddep_launch();
  const uint32_t tmem_base = bars->tmem_base;
  CtaCtl* ctl = &bars->ctl;

  if (warp == 4) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_a);
      auto load_a = [&](int st, int kc) {
        if constexpr (kOut == 4) {
          const SplitWalk w(args.part_chunks, kc);  // a row of the product continues in the matrix's next row
          tma_load_2d(smem + st * kStageBytes, w.a_low() ? &low.a : &tmap_a, &bars->full[st],
                      w.k % args.rows.a_chunks * kBlockK, m0 + w.k / args.rows.a_chunks);
        } else {
          tma_load_2d(smem + st * kStageBytes, &tmap_a, &bars->full[st], kc * kBlockK, m0);
        }
      };
      auto load_w = [&](int st, int kc) {
        if constexpr (kOut == 4) {
          const SplitWalk w(args.part_chunks, kc);
          tma_load_2d(smem + st * kStageBytes + kABytes, w.w_low() ? &low.w : &tmap_w, &bars->full[st], w.k * kBlockK, n0);
        } else {
          tma_load_2d(smem + st * kStageBytes + kABytes, &tmap_w, &bars->full[st], kc * kBlockK, n0);
        }
      };
      const int ahead = args.chunks < kStages ? args.chunks : kStages;
      for (int i = 0; i < ahead; ++i) {
        mbar_arrive_expect_tx(&bars->full[i], kStageBytes);
        load_w(i, chunk0 + i);
      }
      griddep_wait();
      for (int i = 0; i < ahead; ++i) load_a(i, chunk0 + i);
      for (int i = ahead; i < args.chunks; ++i) {
        const int st = i % kStages;
        mbar_wait(&bars->empty[st], (static_cast<uint32_t>(i / kStages) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
        mbar_arrive_expect_tx(&bars->full[st], kStageBytes);
        load_w(st, chunk0 + i);
        load_a(st, chunk0 + i);
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    const bool one = elect_one();
    const int half = two_acc ? args.chunks / 2 : args.chunks;
    for (int i = 0; i < args.chunks; ++i) {
      const int st = i % kStages;
      const uint32_t d_tmem = tmem_base + (i < half ? 0u : static_cast<uint32_t>(kBlockN));
      mbar_wait(&bars->full[st], static_cast<uint32_t>(i / kStages) & 1u, ctl, status, kErrWaitTma);
      tc_fence_after_sync();
      const uint32_t base = smem_u32(smem + st * kStageBytes);
      const uint64_t a_desc = umma_desc_sw128(base);
      const uint64_t b_desc = umma_desc_sw128(base + kABytes);
#pragma unroll
      for (int ks = 0; ks < kBlockK / 16; ++ks)
        if (one) tc_mma_ss(d_tmem, a_desc + 2u * ks, b_desc + 2u * ks, idesc, ((i < half ? i : i - half) | ks) != 0 ? 1u : 0u);
      if (one) tc_commit(&bars->empty[st]);
    }
    if (one) tc_commit(&bars->acc_full);
    __syncwarp();
  }
  griddep_wait();                          // residual and outputs belong to the chain
  // The rows this block owns: rank, rank + S, ... of the tile; eight threads per row, columns 4j.. and 32 + 4j...
  const int n_items = skip ? 0 : n_own * 8;
  auto item_row = [&](int item) { return m0 + ((item >> 3) << log_s) + rank; };
  PieceOperands ops;
  int item = static_cast<int>(threadIdx.x);
  if (item < n_items) load_operands<kOut, kHalves>(args, item_row(item), ntile, item & 7, ops);
  if (warp < 4) {
    mbar_wait(&bars->acc_full, 0, ctl, status, kErrWaitMma);
    tc_fence_after_sync();
  }
  __syncwarp();
  if (split > 1) cluster_wait();           // every block of the cluster runs and has armed its barrier
  if (warp < 4) {
    // Rows grouped by owner in the stage memory (this block's products are complete, nothing else uses it), then one bulk
    // copy per owner.
    const int row = warp * 32 + lane;
    const uint32_t staged = static_cast<uint32_t>((row & (split - 1)) * (kBlockM >> log_s) + (row >> log_s));
    uint8_t* stage = split > 1 ? smem : red;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
#pragma unroll
    for (int h = 0; h < kHalves; ++h) {
      uint32_t v[32];
      tmem_ld32(t_row + h * 32, v);
      tmem_ld_wait();
      if (two_acc) {
        uint32_t other[32];
        tmem_ld32(t_row + kBlockN + h * 32, other);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + __uint_as_float(other[c]));
      }
      if (row < valid) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(stage + red_offset<kBlockN>(staged, h * 8 + c, row)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
    }
    tc_fence_before_sync();
    if (split > 1) {
      fence_proxy_async_smem();
      __syncwarp();
      // this warp's rows of owner `lane`: a contiguous piece of (32 / S) rows, fewer at the end of the matrix
      const int first = warp * (32 >> log_s);
      int rows = ((valid - lane + split - 1) >> log_s) - first;
      if (rows > (32 >> log_s)) rows = 32 >> log_s;
      if (lane < split && rows > 0)
        bulk_copy_to_cta(map_to_cta(smem_u32(red + (rank * (kBlockM >> log_s) + first) * kRowBytes), static_cast<uint32_t>(lane)),
                         smem + (lane * (kBlockM >> log_s) + first) * kRowBytes, static_cast<uint32_t>(rows) * kRowBytes,
                         map_to_cta(smem_u32(&bars->red_full), static_cast<uint32_t>(lane)));
    }
  }
  if (split > 1) {
    if (n_own > 0) mbar_wait_cluster(&bars->red_full, 0, ctl, status, kErrWaitConsumer);
    __syncwarp();
    cluster_arrive();                      // this block's rows are complete; see the end
  } else {
    __syncthreads();
  }

  for (; item < n_items; item += kThreads) {
    const int local = item >> 3, j = item & 7;
    float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < split; ++s) {
      const uint32_t r = s * (kBlockM >> log_s) + local;
      const float4 a = *reinterpret_cast<const float4*>(red + red_offset<kBlockN>(r, j, (local << log_s) + rank));
      lo[0] += a.x; lo[1] += a.y; lo[2] += a.z; lo[3] += a.w;
      if constexpr (kHalves == 2) {
        const float4 b = *reinterpret_cast<const float4*>(red + red_offset<kBlockN>(r, j + 8, (local << log_s) + rank));
        hi[0] += b.x; hi[1] += b.y; hi[2] += b.z; hi[3] += b.w;
      }
    }
    const PieceOperands now = ops;
    if (item + kThreads < n_items) load_operands<kOut, kHalves>(args, item_row(item + kThreads), ntile, (item + kThreads) & 7, ops);
    finish_piece<kOut, VT, kHalves>(args, lo, hi, now, item_row(item), ntile, j, status);
  }

  __syncwarp();
  if (split > 1) cluster_wait();        // every block has its rows: nobody's copies still read this block's memory
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);   // copies that may still be in flight get time to land
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Two blocks fit an SM, so up to two 128 x 64 tiles per SM the grid runs in one wave and a tile's latency is all there is.
// Beyond that the blocks re-read activations and weights too often for what they save, and the 256 x 256 tiles of the
// pair kernels are faster: at K = 512, N = 2048 1024 rows (256 tiles) take 9.1 us here and 10.9 us there, 1500 rows (384
// tiles) 13.9 against 10.9; at K = 2048, N = 512 3678 rows (232 tiles) 17.1 against 22.1, 5000 rows (320) 27.5 against 22.5.
// (Those figures are of the 256 x 256 tiles alone.  Linear layers of more than one tile per SM take half units of the pair kernel where
// those are one wave: fm_linear_gemm.cu.)
bool few_row_tiles(int M, int N) {
  return static_cast<long long>((M + small::kBlockM - 1) / small::kBlockM) * (N / 64) <= 2ll * sm_count();
}

// Blocks per cluster: as many as keep the grid within one block per SM and divide the K chunks.
static int choose_split(int tiles, int k_chunks) {
  int s = 8;
  while (s > 1 && (k_chunks % s != 0 || tiles * s > sm_count())) s >>= 1;
  return s;
}

template <int kOut, typename VT, int kBlockN>
static int launch_tiles(const void* a, const void* w, SmallArgs& args, int K, int in_dtype, int* status,
                        cudaStream_t st, int dependent, const SplitLow* low) {
  using namespace small;
  CUtensorMap tmap_a, tmap_w;
  SplitMaps<kOut == 4> low_maps = {};
  const uint64_t a_rows = kOut == 4 ? static_cast<uint64_t>(low->a_rows) : static_cast<uint64_t>(args.M);
  const uint64_t a_cols = kOut == 4 ? static_cast<uint64_t>(args.rows.a_chunks) * kBlockK : static_cast<uint64_t>(K);
  int rc = encode_rows_16bit(&tmap_a, a, a_rows, a_cols, kBlockM, kBlockK);
  if (rc != 0) return rc;
  rc = encode_rows_16bit(&tmap_w, w, static_cast<uint64_t>(args.N), static_cast<uint64_t>(K), kBlockN, kBlockK);
  if (rc != 0) return rc;
  const int m_tiles = (args.M + kBlockM - 1) / kBlockM, n_tiles = args.N / kBlockN;
  if constexpr (kOut == 4) {
    rc = encode_rows_16bit(&low_maps.a, low->a, a_rows, a_cols, kBlockM, kBlockK);
    if (rc == 0) rc = encode_rows_16bit(&low_maps.w, low->w, static_cast<uint64_t>(args.N), static_cast<uint64_t>(K), kBlockN, kBlockK);
    if (rc != 0) return rc;
  }
  if constexpr (kOut == 4) args.part_chunks = K / kBlockK / args.rows.parts;
  const int k_chunks = (kOut == 4 ? 3 : 1) * (K / kBlockK);
  args.split = choose_split(m_tiles * n_tiles, k_chunks);
  args.chunks = k_chunks / args.split;
  const int fmt = in_dtype == 1 ? 0 : 1;
  const uint32_t idesc = umma_idesc_f16(kBlockM, kBlockN, fmt, fmt, 0, 0);
  auto kern = linear_small_kernel<kOut, VT, kBlockN>;
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), Tile<kBlockN>::kSmemBytes);
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(n_tiles * args.split, m_tiles), kThreads, Tile<kBlockN>::kSmemBytes, st, args.split, dependent, tmap_a,
                       tmap_w, low_maps, args, idesc, status);
}

// 64-column tiles, or 32 where 64 would leave the K split at its limit of eight with SMs to spare: the partial sums that
// cross the cluster are what a split costs (28 KB out of and into every block at eight blocks of 64 columns, about 1.9 us;
// 14 KB with 32), and halving the tile halves them.
template <int kOut, typename VT>
static int launch_small(const void* a, const void* w, SmallArgs& args, int K, int in_dtype, int* status, cudaStream_t st,
                        int dependent, const SplitLow* low = nullptr) {
  if constexpr (kOut != 3) {
    if (static_cast<long long>((args.M + 127) / 128) * (args.N / 64) * 8 <= sm_count())
      return launch_tiles<kOut, VT, 32>(a, w, args, K, in_dtype, status, st, dependent, low);
  }
  return launch_tiles<kOut, VT, 64>(a, w, args, K, in_dtype, status, st, dependent, low);
}

int launch_linear_small(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N, int K,
                        int in_dtype, int out_dtype, int gelu, int* status, cudaStream_t st, int dependent) {
  SmallArgs args = {};
  args.scale = scale;
  args.resid = resid;
  args.y = y;
  args.M = M;
  args.N = N;
  args.gelu = gelu;
  if (out_dtype == 2) return launch_small<2, __half>(a, w, args, K, in_dtype, status, st, dependent);
  if (out_dtype == 1) return launch_small<1, __half>(a, w, args, K, in_dtype, status, st, dependent);
  return launch_small<0, __half>(a, w, args, K, in_dtype, status, st, dependent);
}

int launch_linear_split_small(const void* a_hi, const void* w_hi, const SplitLow& low, const SplitRows& map, float* y, int M, int N,
                              int K, int* status, cudaStream_t st, int dependent) {
  SmallArgs args = {};
  args.y = y;
  args.M = M;
  args.N = N;
  args.rows = map;
  return launch_small<4, __half>(a_hi, w_hi, args, K, 1, status, st, dependent, &low);
}

int launch_qkv_small(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status,
                     cudaStream_t st, int dependent) {
  SmallArgs args = {};
  args.M = M;
  args.N = 1536;
  args.qkv = ep;
  const int in_dtype = (dtype_flags & 2) ? 1 : 0;
  if (dtype_flags & 1) return launch_small<3, __half>(x, w_qkv, args, 512, in_dtype, status, st, dependent);
  return launch_small<3, __nv_bfloat16>(x, w_qkv, args, 512, in_dtype, status, st, dependent);
}

}  // namespace fm
