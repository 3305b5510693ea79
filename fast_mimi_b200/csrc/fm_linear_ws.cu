// Linear layers for a few hundred rows with the weights resident in tensor memory (sm_100a): y = residual + scale * act(a W^T),
// K = 512 .. 4096 in slices of 512.
//
// Latency-bound, like fm_linear_small.cu, whose blocks of 128 rows x 64 (32) outputs fetch the rows of their slice of K after the wait
// for the kernel in front, 64 KB and more, and share K eight ways.  Here a block owns 128 outputs x 16 to 128 rows and 512 of K:
// its weights, 128 KB, go by way of shared memory into tensor memory (the A operand, 256 columns) ahead of the wait, and what
// it fetches behind it is kRows KB.  The blocks of a cluster share K; rows kRows / S r .. of the tile belong to cluster rank r, every block
// sends its FP32 partial sums of an owner's rows with one bulk copy, and the owner adds them in rank order (the result does not
// depend on timing), applies the epilogue and stores whole lines.
//
// A call by itself, few-row kernel (or half units of the pair kernel) -> this one, us, FP32 residual: K = 512, N = 512 1 row 4.8 -> 4.4, 128 rows 5.9 -> 4.8,
// 400 7.1 -> 5.2, 1000 7.9 -> 6.1, 2368 7.6 -> 6.8; K = 2048, N = 512 1 row 6.5 -> 5.1, 128 7.0 -> 6.0, 400 8.3 -> 7.7; K = 512, N = 2048 with GELU 128 rows 7.3 ->
// 5.5, 576 8.2 -> 7.2.  GPU time of eight layers (o_proj, and to 512 rows fc2): a clip of 190 frames 207 -> 187 us, four of 125 260 -> 216, eight 331 -> 317;
// 250 live streams 378 -> 353, five of 50 frames 252 -> 230, ten of 30 284 -> 236.
//
// Sixteen warps: weights, accumulator and epilogue.  Warp 0 also asks for the rows and issues the products.
#include "fm_device_fact.h"
#include "fm_launch.h"
#include "fm_small_tile.cuh"

namespace fm {

namespace ws {
constexpr int kSlice = 512, kBlockN = 128, kChunks = kSlice / 64;
constexpr int kWBox = kBlockN * 128, kWBytes = kChunks * kWBox;      // 64 of K; a block's weights
constexpr int kWarps = 16, kThreads = kWarps * 32, kMaxSplit = 8;
constexpr int kTmemCols = 512, kTmemD = kSlice / 2;                  // weights | accumulators
constexpr int kOutRow = kBlockN * 4;                                 // bytes of a row of results
constexpr int kQuarters = 4;                                         // of a block's rows' K, loaded and waited for one by one where a block has 128
struct Barriers {
  uint64_t w_full;
  uint64_t a_full[kQuarters];
  uint64_t acc_full;
  uint64_t red_full;         // the partial sums of this block's rows have arrived from every block of the cluster
  uint32_t tmem_base;
  CtaCtl ctl;
};
// Up to 64 rows: weights, later this block's partial sums (first half) and those that it is sent (second half) | rows.  128 rows: weights, later
// the rows, later this block's partial sums | those that it is sent
constexpr int smem_bytes(int rows) { return 1024 + kWBytes + (rows == 128 ? 128 * kOutRow : kChunks * rows * 128) + static_cast<int>(sizeof(Barriers)); }
static_assert(smem_bytes(64) <= 232448 && smem_bytes(128) <= 232448 && 64 * kOutRow <= kWBytes / 2, "exceeds the 227 KB a block may use");

__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
}  // namespace ws

// kOut: 0 = BF16, 1 = FP16, 2 = FP32 output and residual; 3 = q | k | v with RoPE (VT: type of v)
template <int kOut, typename VT, int kRows>
__global__ void __launch_bounds__(ws::kThreads, 1)
linear_ws_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ SmallArgs args,
                 uint32_t idesc, int* status) {
  using namespace ws;
  constexpr int kItems = (kRows * 16 + kThreads - 1) / kThreads;       // pieces of eight results of a thread
  // accumulators of 64, 128 or 256 of K each, added up in FP32: in one of 512 the tensor core cuts more of the addends (3.2e-7 of the result instead of 1e-7,
  // with a residual as large as the product; 6.5e-7 and 1.9e-7 of the product alone).
  // q | k | v of 128 rows a block, which a layer's chain alone takes, are one all the same: so they are in the kernels that fewer or more rows take there, and what
  // a stream's ring holds must not depend on how many others share its calls.
  constexpr int kSums = kRows == 16 ? 8 : (kRows == 128 ? (kOut == 3 ? 1 : 2) : 4), kPer = kChunks / kSums;
  constexpr bool kTall = kRows == 128;
  constexpr int kParts = kTall ? kQuarters : 1;                        // of the rows' K, a barrier each
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_w = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = kTall ? smem_w : smem_w + kWBytes;
  uint8_t* red = kTall ? smem_w + kWBytes : smem_w + kWBytes / 2;
  Barriers* bars = reinterpret_cast<Barriers*>(smem_w + kWBytes + (kTall ? 128 * kOutRow : kChunks * kRows * 128));
  CtaCtl* ctl = &bars->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = args.split;
  const int rank = split > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int ntile = static_cast<int>(blockIdx.x) / split;
  const int m0 = static_cast<int>(blockIdx.y) * kRows;
  const int own = kRows / split;                                       // rows of an owner
  const uint32_t slab = static_cast<uint32_t>(own) * kOutRow;
  // read early: a status set before this chain began stops every kernel of it (the stores are left out)
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  if (threadIdx.x == 0) {
    mbar_init(&bars->w_full, 1);
    for (int i = 0; i < kParts; ++i) mbar_init(&bars->a_full[i], 1);
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->red_full, 1);
    ctl->abort = 0;
    fence_mbar_init();
    if (split > 1) mbar_arrive_expect_tx(&bars->red_full, static_cast<uint32_t>(split) * slab);
    mbar_arrive_expect_tx(&bars->w_full, kWBytes);
#pragma unroll
    for (int kc = 0; kc < kChunks; ++kc) tma_load_2d(smem_w + kc * kWBox, &tmap_w, &bars->w_full, rank * kSlice + kc * 64, ntile * kBlockN);
    tma_prefetch_desc(&tmap_a);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  griddep_launch();
  const uint32_t tmem_base = bars->tmem_base, t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);

  // Weights: output 32 (warp % 4) + lane, two values of K a column
  mbar_wait(&bars->w_full, 0, ctl, status, kErrWaitTma);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int kc = 2 * (warp >> 2) + i;
    uint32_t r[32];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const uint4 v = *reinterpret_cast<const uint4*>(smem_w + kc * kWBox + sw128_offset((warp & 3) * 32 + lane, p));
      r[4 * p] = v.x; r[4 * p + 1] = v.y; r[4 * p + 2] = v.z; r[4 * p + 3] = v.w;
    }
    tmem_st32(t_row + kc * 32, r);
  }
  tmem_st_wait();
  tc_fence_before_sync();
  if (kTall || split > 1) fence_proxy_async_smem();        // the rows, or other blocks' copies, come where the weights were read
  __syncthreads();                         // the weights are in tensor memory, and the place where they lay is free
  if (split > 1) cluster_arrive_relaxed();
  griddep_wait();

  if (warp == 0) {
    tc_fence_after_sync();
    const bool one = elect_one();
    if (one) {
#pragma unroll
      for (int part = 0; part < kParts; ++part) {
        mbar_arrive_expect_tx(&bars->a_full[part], kChunks / kParts * kRows * 128);
#pragma unroll
        for (int kc = part * kChunks / kParts; kc < (part + 1) * kChunks / kParts; ++kc)
          tma_load_2d(smem_a + kc * kRows * 128, &tmap_a, &bars->a_full[part], rank * kSlice + kc * 64, m0);
      }
    }
    __syncwarp();
    const uint64_t rows = umma_desc_sw128(smem_u32(smem_a));
    auto arrived = [&](int part) {
      mbar_wait(&bars->a_full[part], 0, ctl, status, kErrWaitTma);
      __syncwarp();
      tc_fence_after_sync();
    };
    if constexpr (kParts == 1) arrived(0);
    for (int kc = 0; kc < kChunks; ++kc) {
      if constexpr (kParts > 1) {
        if (kc % (kChunks / kParts) == 0) arrived(kc / (kChunks / kParts));
      }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (one)
          tc_mma_ts(tmem_base + kTmemD + kc / kPer * kRows, tmem_base + kc * 32 + ks * 8, rows + static_cast<uint64_t>(kc * kRows * 128 >> 4) + 2u * ks,
                    idesc, (kc % kPer | ks) != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&bars->acc_full);
    __syncwarp();
  }
  // item: row item / 16 of those this block owns, half (item / 8) % 2 of its columns, piece item % 8
  const int first = m0 + rank * own, n_own = args.M - first < own ? args.M - first : own;
  const int n_items = skip ? 0 : n_own * 16;
  // what the epilogue reads besides, asked for two pieces a thread ahead
  constexpr int kAhead = kItems < 2 ? kItems : 2;
  PieceOperands ops[kAhead];
  auto item_of = [&](int i) { return static_cast<int>(threadIdx.x) + i * kThreads; };
  auto ask = [&](int i) {
    const int item = item_of(i);
    if (item < n_items) load_operands<kOut>(args, first + (item >> 4), 2 * ntile + ((item >> 3) & 1), item & 7, ops[i % kAhead]);
  };
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ask(i);
  mbar_wait(&bars->acc_full, 0, ctl, status, kErrWaitMma);
  __syncwarp();
  tc_fence_after_sync();
  {
    // output 32 (warp % 4) + lane, a quarter of the rows a warp
    constexpr int kN = kRows / 4;
    float sum[kN];
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      uint32_t u[kN];
      const uint32_t at = t_row + kTmemD + k * kRows + (warp >> 2) * kN;
      if constexpr (kN == 4) tmem_ld4(at, u);
      else if constexpr (kN == 8) tmem_ld8(at, u);
      else if constexpr (kN == 16) tmem_ld16(at, u);
      else tmem_ld32(at, u);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kN; ++i) sum[i] = k == 0 ? __uint_as_float(u[i]) : sum[i] + __uint_as_float(u[i]);
    }
#pragma unroll
    for (int i = 0; i < kN; ++i) reinterpret_cast<float*>(smem_w)[((warp >> 2) * kN + i) * kBlockN + (warp & 3) * 32 + lane] = sum[i];
    tc_fence_before_sync();
  }
  if (split > 1) {
    fence_proxy_async_smem();
    __syncthreads();
    cluster_wait();                        // every block of the cluster runs, and its memory is free
    if (warp < split && lane == 0)
      asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(map_to_cta(smem_u32(red + rank * slab), static_cast<uint32_t>(warp))), "r"(smem_u32(smem_w + warp * slab)), "r"(slab),
                   "r"(map_to_cta(smem_u32(&bars->red_full), static_cast<uint32_t>(warp))) : "memory");
    __syncwarp();
    mbar_wait_cluster(&bars->red_full, 0, ctl, status, kErrWaitConsumer);
    __syncwarp();
    cluster_arrive_relaxed();              // this block's rows are complete; see the end
  } else {
    __syncthreads();
  }
  const uint8_t* sums = split > 1 ? red : smem_w;
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int item = item_of(i);
    const PieceOperands now = ops[i % kAhead];
    if (i + kAhead < kItems) ask(i + kAhead);
    if (item < n_items) {
      const int local = item >> 4, sub = (item >> 3) & 1, j = item & 7;
      float lo[4] = {0.f, 0.f, 0.f, 0.f}, hi[4] = {0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < split; ++s) {
        const uint8_t* row = sums + s * slab + local * kOutRow + sub * 256 + j * 16;
        const float4 a = *reinterpret_cast<const float4*>(row), b = *reinterpret_cast<const float4*>(row + 128);
        lo[0] += a.x; lo[1] += a.y; lo[2] += a.z; lo[3] += a.w;
        hi[0] += b.x; hi[1] += b.y; hi[2] += b.z; hi[3] += b.w;
      }
      finish_piece<kOut, VT>(args, lo, hi, now, first + local, 2 * ntile + sub, j, status);
    }
  }
  if (split > 1) {
    __syncwarp();
    cluster_wait();                        // every block has its rows: nobody's copies still read this block's memory
  }
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);      // copies that may still be in flight get time to land
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

static long long blocks_for(int M, int N, int K, int rows) {
  return static_cast<long long>((M + rows - 1) / rows) * (N / ws::kBlockN) * (K / ws::kSlice);
}
namespace {
// Clusters of so many blocks that the device runs at once (a block has an SM); 0: none, or not to be found out just now.
int clusters_of(int split) {
  static DeviceFact known[4];
  int dev = 0, at = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  while (1 << at < split) ++at;
  const int n = known[at].get(dev, [split] {
    const auto kern = linear_ws_kernel<2, __half, 64>;
    return ensure_dynamic_smem(reinterpret_cast<const void*>(kern), ws::smem_bytes(64)) == 0 ? resident_clusters(kern, ws::kThreads, ws::smem_bytes(64), split)
                                                                                             : -1;
  });
  return n > 0 ? n : 0;
}
}  // namespace

// Rows of a block, 0: not a call for this kernel.  In a chain as few as leave half of the SMs to the kernels in front and behind, whose
// blocks then bring their weights while this one runs, by itself as few as a block per SM allows; 64 up to a block per SM, as far as the
// device holds the clusters at once (K = 2048, N = 512: 512 rows 8.0 us, 528 in two waves 12.5 where the other kernel takes 10.2; K = 4096 128 rows 10.8
// and 8.0).  A second tile of 64 with few rows in it is not worth one (K = N = 2048, 72 rows 7.9 us, 7.6 there).  Nor are two blocks that share K for 256 outputs and
// one tile of the other kernel, where eight do (K = 1024, N = 256 1 row 4.6 to 4.8 us there, 5.1 here, 64 rows 5.0 and 5.2, 128 5.3 and 5.3, 144 5.8 and 5.3; N = 512 1 row
// 5.4 and 5.1).
// 128 rows, whose loads follow the weights into the same memory, by themselves are no faster than the other kernels (K = 2048, N = 512
// 640 rows 9.9 -> 10.1 us; K = 512, N = 2048 with GELU 8.2 -> 8.9).  In a chain, where the weights come early, they are: with K shared by four or
// more, and, without, as far as two thirds of the SMs (eight layers of five clips of 125 frames 278 -> 268 -> 260 us, of 577 BF16 frames 302 -> 291 ->
// 279; beyond, eight clips 306 -> 314).  Not for up to 512 outputs onto a residual of 16 bits, 2369 rows and more, where half units of the pair kernel take 48 pairs of blocks
// at once (eight layers of 14 clips of 170 BF16 frames, there and here, 416 and 422, of 200 422 and 428; FP32 416 and 416, 422 and 421).
static int rows_per_block(int M, int N, int K, int dependent, bool resid16) {
  const int split = K / ws::kSlice;
  if (M <= 0 || N % ws::kBlockN != 0 || K % ws::kSlice != 0 || split > ws::kMaxSplit || (split & (split - 1)) != 0) return 0;
  if (split == 2 && N == 2 * ws::kBlockN && M <= 128) return 0;
  const int clusters = clusters_of(split);
  for (int rows = 16; rows <= 128; rows *= 2) {
    const long long blocks = blocks_for(M, N, K, rows), room = dependent && rows < 64 ? sm_count() / 2 : sm_count();
    if (rows == 128 && (!dependent || (split == 1 ? 3 * blocks > 2 * sm_count() || (resid16 && N <= 4 * ws::kBlockN) : split < 4))) return 0;
    if (blocks <= room && blocks / split <= clusters) return rows >= 64 && M > rows && M <= rows * 3 / 2 ? 0 : rows;
  }
  return 0;
}

bool linear_ws_takes(int M, int N, int K, int dependent, bool resid16) { return rows_per_block(M, N, K, dependent, resid16) != 0; }

// a [M, K] and w [N, K]: the launch of one of the kernels for 16, 32, 64 and 128 rows a block
using Kern = void (*)(const CUtensorMap, const CUtensorMap, const SmallArgs, uint32_t, int*);
static int launch_ws(const Kern (&kerns)[4], const void* a, const void* w, SmallArgs& args, int rows, int K, int in_dtype, int* status, cudaStream_t st,
                     int dependent) {
  using namespace ws;
  args.split = K / kSlice;
  const int fmt = in_dtype == 1 ? 0 : 1;
  CUtensorMap tmap_a, tmap_w;
  int rc = encode_rows_16bit(&tmap_a, a, static_cast<uint64_t>(args.M), static_cast<uint64_t>(K), static_cast<uint32_t>(rows), 64);
  if (rc == 0) rc = encode_rows_16bit(&tmap_w, w, static_cast<uint64_t>(args.N), static_cast<uint64_t>(K), kBlockN, 64);
  if (rc != 0) return rc;
  const Kern kern = kerns[rows == 16 ? 0 : rows == 32 ? 1 : rows == 64 ? 2 : 3];
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes(rows));
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(args.N / kBlockN * args.split, (args.M + rows - 1) / rows), kThreads, smem_bytes(rows), st, args.split, dependent, tmap_a,
                       tmap_w, args, umma_idesc_f16(128, rows, fmt, fmt, 0, 0), status);
}

int launch_linear_ws(const void* a, const void* w, void* y, ParamVec scale, const void* resid, int M, int N, int K, int in_dtype, int out_dtype, int gelu,
                     int* status, cudaStream_t st, int dependent) {
  const int rows = rows_per_block(M, N, K, dependent, resid != nullptr && out_dtype != 2);
  if (rows == 0) return -1;
  SmallArgs args = {};
  args.scale = scale;
  args.resid = resid;
  args.y = y;
  args.M = M;
  args.N = N;
  args.gelu = gelu;
  static const Kern table[3][4] = {
      {linear_ws_kernel<0, __half, 16>, linear_ws_kernel<0, __half, 32>, linear_ws_kernel<0, __half, 64>, linear_ws_kernel<0, __half, 128>},
      {linear_ws_kernel<1, __half, 16>, linear_ws_kernel<1, __half, 32>, linear_ws_kernel<1, __half, 64>, linear_ws_kernel<1, __half, 128>},
      {linear_ws_kernel<2, __half, 16>, linear_ws_kernel<2, __half, 32>, linear_ws_kernel<2, __half, 64>, linear_ws_kernel<2, __half, 128>}};
  return launch_ws(table[out_dtype], a, w, args, rows, K, in_dtype, status, st, dependent);
}

int launch_qkv_ws(const void* x, const void* w_qkv, const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status, cudaStream_t st, int dependent) {
  using bf16 = __nv_bfloat16;
  const int rows = rows_per_block(M, 1536, 512, dependent, false);
  if (rows == 0) return -1;
  SmallArgs args = {};
  args.M = M;
  args.N = 1536;
  args.qkv = ep;
  static const Kern table[2][4] = {
      {linear_ws_kernel<3, bf16, 16>, linear_ws_kernel<3, bf16, 32>, linear_ws_kernel<3, bf16, 64>, linear_ws_kernel<3, bf16, 128>},
      {linear_ws_kernel<3, __half, 16>, linear_ws_kernel<3, __half, 32>, linear_ws_kernel<3, __half, 64>, linear_ws_kernel<3, __half, 128>}};
  return launch_ws(table[dtype_flags & 1], x, w_qkv, args, rows, 512, (dtype_flags & 2) ? 1 : 0, status, st, dependent);
}

}  // namespace fm
