// LayerNorm and the product behind it in one kernel, for few rows (sm_100a):  q | k | v with RoPE, or gelu(.),  of
// LayerNorm(x) W^T with 512 channels.  Reference: src/fast_mimi/model.py:2021-2024 with :1897-1912 and :1990-1999.
//
// Latency-bound: at one clip's rows a LayerNorm launch (1.5 us of memory round trip and reductions) and the product
// behind it (2.5 us) each pay a kernel boundary.  Here a block owns `kRows` rows (16, 32 or 64) x 128 outputs (two heads).  Its sixteen
// warps bring the whole K = 512 of its weight slice (128 KB) by way of shared memory into tensor memory, where it is the A operand (256
// columns), ahead of the wait for the kernel in front; then they normalise the rows, up to four a warp, straight into the swizzled other
// operand.  There is no K split, hence no cluster and no reduction.  Every block repeats the normalisation of its rows (2 KB of x a row from
// L2), which is what limits the rows.
//
// With weights as the 128 rows of the product and in tensor memory an instruction takes 19 cycles for 16 columns and 32 for 64; with
// rows as its rows, both operands in shared memory and waits between them, it took 75.  GPU time of eight layers, from the kernel that
// did that (16 or 32 rows x 64 outputs, to 160 rows; beyond, a LayerNorm kernel and fm_linear_small.cu) to this one, us: clip of 17 frames 98 -> 92, 125 frames
// 160 -> 158, two clips of 125 252 -> 217, four 290 -> 258, six 329 -> 310; 190 streams of one frame 347 -> 312, 384 519 -> 476; five of 50 frames 290 -> 252.
// Tried: several row tiles one after another in a block, for more rows: 250 rows 217 -> 238, 1000 rows in two turns 331 -> 387.
//
// Warps 0-15: weights, LayerNorm, accumulator and epilogue.  Warp 0 also issues the products.
#include <type_traits>

#include "fm_launch.h"
#include "fm_small_tile.cuh"

namespace fm {

namespace lnlin {
constexpr int kHidden = 512;
constexpr int kBlockN = 128;
constexpr int kChunks = kHidden / 64;
constexpr int kWBox = kBlockN * 128, kWBytes = kChunks * kWBox;      // 64 of K; the weight slice
constexpr int kWarps = 16, kThreads = kWarps * 32;
constexpr int kTmemCols = 512, kTmemD = kHidden / 2;                 // weights | accumulators
struct Barriers {
  uint64_t w_full;
  uint64_t acc_full;
  uint32_t tmem_base;
  CtaCtl ctl;
};
// Weights, later the results in FP32 | LayerNorm's result
constexpr int smem_bytes(int rows) { return 1024 + kWBytes + kChunks * rows * 128 + static_cast<int>(sizeof(Barriers)); }
static_assert(smem_bytes(64) <= 232448, "exceeds the 227 KB a block may use");
}  // namespace lnlin

struct LnArgs {
  const void* x;          // [M, 512]
  ParamVec weight;
  ParamVec bias;
  float eps;
  int x_type;             // 0 BF16, 1 FP16, 2 FP32
  int opens_chain;        // first kernel of a chain: lets the next one start only after its own wait
};

// kTc: type of the product's operands (0 BF16, 1 FP16); kOut: kTc, or 3 = q | k | v
template <int kTc, int kOut, typename VT, int kRows>
__global__ void __launch_bounds__(lnlin::kThreads, 1)
ln_linear_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ LnArgs ln,
                 const __grid_constant__ SmallArgs args, uint32_t idesc, int* status) {
  using namespace lnlin;
  using TOp = typename std::conditional<kTc == 1, __half, __nv_bfloat16>::type;
  constexpr int kMine = kRows / kWarps;                  // rows of a warp
  constexpr int kItems = (kRows * 16 + kThreads - 1) / kThreads;       // pieces of eight results of a thread
  // 256 of K in an accumulator, added up in FP32 (FP16 operands, FP32 results against 64 bits: one of 512 6.5e-7, two 3.4e-7, four 1.9e-7; clip of 125 frames,
  // five streams of 50 frames, eight layers: the same time within 0.5 %).  q | k | v are one all the same, as in every kernel of a layer's call that makes
  // them: a ring's bits must not depend on which of them did.
  constexpr int kSums = kOut == 3 ? 1 : 2, kPer = kChunks / kSums;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_w = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_h = smem_w + kWBytes;
  float* smem_o = reinterpret_cast<float*>(smem_w);
  Barriers* bars = reinterpret_cast<Barriers*>(smem_h + kChunks * kRows * 128);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = static_cast<int>(blockIdx.x) * kBlockN;
  const int m0 = static_cast<int>(blockIdx.y) * kRows;
  // read early: a status set before this chain began stops every kernel of it (the stores are left out)
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  if (threadIdx.x == 0) {
    mbar_init(&bars->w_full, 1);
    mbar_init(&bars->acc_full, 1);
    bars->ctl.abort = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&bars->w_full, kWBytes);
#pragma unroll
    for (int kc = 0; kc < kChunks; ++kc) tma_load_2d(smem_w + kc * kWBox, &tmap_w, &bars->w_full, kc * 64, n0);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (!ln.opens_chain) griddep_launch();
  const uint32_t tmem_base = bars->tmem_base, t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  CtaCtl* ctl = &bars->ctl;
  const int n_rows = args.M - m0 < kRows ? args.M - m0 : kRows;

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
  tc_fence_before_sync();                  // the products follow behind a barrier of the block
  griddep_wait();
  if (ln.opens_chain) griddep_launch();

  // ---- LayerNorm.  This lane's channels: 4 * lane + 128 * j + (0..3)
  {
    float v[kMine][4][4];
    uint4 w_raw[4], b_raw[4];
    auto params = [&](auto f32) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w_raw[j] = ln.weight.raw4<decltype(f32)::value>(128 * j + 4 * lane);
        b_raw[j] = ln.bias.raw4<decltype(f32)::value>(128 * j + 4 * lane);
      }
    };
    if (ln.x_type == 2) {
#pragma unroll
      for (int i = 0; i < kMine; ++i) {
        const int r = i * kWarps + warp < n_rows ? i * kWarps + warp : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) load4<2>(ln.x, static_cast<long long>(m0 + r) * kHidden + 128 * j + 4 * lane, v[i][j]);
      }
      params(std::true_type());
    } else {
      uint2 u[kMine][4];
#pragma unroll
      for (int i = 0; i < kMine; ++i) {
        const int r = i * kWarps + warp < n_rows ? i * kWarps + warp : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          u[i][j] = __ldcg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(ln.x) + static_cast<long long>(m0 + r) * kHidden + 128 * j + 4 * lane));
      }
      params(std::false_type());
#pragma unroll
      for (int i = 0; i < kMine; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 lo = ln.x_type == 1 ? Pack16<__half>::unpack(u[i][j].x) : Pack16<__nv_bfloat16>::unpack(u[i][j].x);
          const float2 hi = ln.x_type == 1 ? Pack16<__half>::unpack(u[i][j].y) : Pack16<__nv_bfloat16>::unpack(u[i][j].y);
          v[i][j][0] = lo.x; v[i][j][1] = lo.y; v[i][j][2] = hi.x; v[i][j][3] = hi.y;
        }
      }
    }
    // the same sums in the same order as layernorm512_kernel
    float sum[kMine], sq[kMine];
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      sum[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i] += (v[i][j][0] + v[i][j][1]) + (v[i][j][2] + v[i][j][3]);
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
    float w[4][4], b[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 wf = ln.x_type == 2 ? ln.weight.value4<true>(w_raw[j]) : ln.weight.value4(w_raw[j]);
      const float4 bf = ln.x_type == 2 ? ln.bias.value4<true>(b_raw[j]) : ln.bias.value4(b_raw[j]);
      w[j][0] = wf.x; w[j][1] = wf.y; w[j][2] = wf.z; w[j][3] = wf.w;
      b[j][0] = bf.x; b[j][1] = bf.y; b[j][2] = bf.z; b[j][3] = bf.w;
    }
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int r = i * kWarps + warp;
      const float rstd = rsqrtf(sq[i] * (1.0f / kHidden) + ln.eps);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = v[i][j][e] * rstd * w[j][e] + b[j][e];
        // channels 128 j + 4 lane ..: chunk 2 j + lane / 16, 16-byte piece (lane % 16) / 2, its lower or upper half
        uint8_t* dst = smem_h + (2 * j + (lane >> 4)) * (kRows * 128) + sw128_offset(r, (lane & 15) >> 1) + (lane & 1) * 8;
        *reinterpret_cast<uint2*>(dst) = make_uint2(Pack16<TOp>::pack(o[0], o[1]), Pack16<TOp>::pack(o[2], o[3]));
      }
    }
    fence_proxy_async_smem();
  }
  __syncthreads();                         // the operand is complete, and the weights are in tensor memory

  if (warp == 0) {
    tc_fence_after_sync();
    const uint64_t h = umma_desc_sw128(smem_u32(smem_h));
    const bool one = elect_one();
    for (int kc = 0; kc < kChunks; ++kc) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (one)
          tc_mma_ts(tmem_base + kTmemD + kc / kPer * kRows, tmem_base + kc * 32 + ks * 8, h + static_cast<uint64_t>(kc * kRows * 128 >> 4) + 2u * ks, idesc,
                    (kc % kPer | ks) != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&bars->acc_full);
    __syncwarp();
  }
  // item: row item / 16 of the block, head (item / 8) % 2, piece item % 8
  const int n_items = skip ? 0 : n_rows * 16;
  PieceOperands ops[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int item = static_cast<int>(threadIdx.x) + i * kThreads;
    if (item < n_items) load_operands<kOut>(args, m0 + (item >> 4), 2 * static_cast<int>(blockIdx.x) + ((item >> 3) & 1), item & 7, ops[i]);
  }
  mbar_wait(&bars->acc_full, 0, ctl, status, kErrWaitMma);
  __syncwarp();
  tc_fence_after_sync();
  {
    // output 32 (warp % 4) + lane, a quarter of the rows a warp
    constexpr int kN = kRows / 4;
    uint32_t u[kSums][kN];
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      const uint32_t at = t_row + kTmemD + k * kRows + (warp >> 2) * kN;
      if constexpr (kN == 4) tmem_ld4(at, u[k]);
      else if constexpr (kN == 8) tmem_ld8(at, u[k]);
      else tmem_ld16(at, u[k]);
    }
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      float sum = __uint_as_float(u[0][i]);
      if constexpr (kSums == 2) sum += __uint_as_float(u[1][i]);
      smem_o[((warp >> 2) * kN + i) * kBlockN + (warp & 3) * 32 + lane] = sum;
    }
    tc_fence_before_sync();
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int item = static_cast<int>(threadIdx.x) + i * kThreads;
    if (item < n_items) {
      const int local = item >> 4, sub = (item >> 3) & 1, j = item & 7;
      const float* row = smem_o + local * kBlockN + sub * 64 + 4 * j;
      const float4 a = *reinterpret_cast<const float4*>(row), c = *reinterpret_cast<const float4*>(row + 32);
      float lo[4] = {a.x, a.y, a.z, a.w}, hi[4] = {c.x, c.y, c.z, c.w};
      finish_piece<kOut, VT>(args, lo, hi, ops[i], m0 + local, 2 * static_cast<int>(blockIdx.x) + sub, j, status);
    }
  }
  if (ctl->abort) __nanosleep(20000);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

static long long blocks_for(int M, int N, int rows) { return static_cast<long long>((M + rows - 1) / rows) * (N / lnlin::kBlockN); }
// As few rows as leave half of the SMs to the kernels in front and behind, whose blocks then bring their weights while this one runs; 64 up to
// a block per SM (768 rows of q | k | v, 576 of an MLP of 2048).  Beyond that the separate kernels are faster (see above).
static int rows_per_block(int M, int N) {
  int rows = 16;
  while (rows < 64 && 2 * blocks_for(M, N, rows) > sm_count()) rows *= 2;
  return rows;
}

bool few_rows_with_norm(int M, int N) { return N % lnlin::kBlockN == 0 && blocks_for(M, N, 64) <= sm_count(); }

template <int kTc, int kOut, typename VT>
static int launch_rows(const CUtensorMap& tmap_w, const LnArgs& ln, const SmallArgs& args, int* status, cudaStream_t st, int dependent) {
  using namespace lnlin;
  const int rows = rows_per_block(args.M, args.N), fmt = kTc == 1 ? 0 : 1;
  auto kern = rows == 16 ? ln_linear_kernel<kTc, kOut, VT, 16> : rows == 32 ? ln_linear_kernel<kTc, kOut, VT, 32> : ln_linear_kernel<kTc, kOut, VT, 64>;
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes(rows));
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(args.N / kBlockN, (args.M + rows - 1) / rows), kThreads, smem_bytes(rows), st, 1, dependent,
                       tmap_w, ln, args, umma_idesc_f16(128, rows, fmt, fmt, 0, 0), status);
}

static int launch_ln(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, const void* w,
                     const SmallArgs& args, int tc_fp16, int qkv, int value_fp16, int opens_chain, int* status, cudaStream_t st,
                     int dependent) {
  if (x_dtype < 0 || x_dtype > 2 || args.M <= 0 || args.N % lnlin::kBlockN != 0) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight.data) | reinterpret_cast<uintptr_t>(bias.data) |
       reinterpret_cast<uintptr_t>(w)) & 15u)
    return -3;
  CUtensorMap tmap_w;
  const int rc = encode_rows_16bit(&tmap_w, w, static_cast<uint64_t>(args.N), lnlin::kHidden, lnlin::kBlockN, 64);
  if (rc != 0) return rc;
  const LnArgs ln = {x, weight, bias, eps, x_dtype, opens_chain};
  if (tc_fp16) {
    if (!qkv) return launch_rows<1, 1, __half>(tmap_w, ln, args, status, st, dependent);
    return value_fp16 ? launch_rows<1, 3, __half>(tmap_w, ln, args, status, st, dependent)
                      : launch_rows<1, 3, __nv_bfloat16>(tmap_w, ln, args, status, st, dependent);
  }
  if (!qkv) return launch_rows<0, 0, __half>(tmap_w, ln, args, status, st, dependent);
  return value_fp16 ? launch_rows<0, 3, __half>(tmap_w, ln, args, status, st, dependent)
                    : launch_rows<0, 3, __nv_bfloat16>(tmap_w, ln, args, status, st, dependent);
}

int launch_ln_qkv(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, const void* w_qkv,
                  const QkvEpilogueArgs& ep, int M, int dtype_flags, int* status, cudaStream_t st, int dependent) {
  SmallArgs args = {};
  args.M = M;
  args.N = 1536;
  args.qkv = ep;
  return launch_ln(x, x_dtype, weight, bias, eps, w_qkv, args, (dtype_flags & 2) ? 1 : 0, 1, dtype_flags & 1, 1, status, st,
                   dependent);
}

int launch_ln_linear_gelu(const void* x, int x_dtype, ParamVec weight, ParamVec bias, float eps, const void* w, void* y,
                          int M, int N, int tc_fp16, int* status, cudaStream_t st, int dependent) {
  SmallArgs args = {};
  args.y = y;
  args.M = M;
  args.N = N;
  args.gelu = 1;
  return launch_ln(x, x_dtype, weight, bias, eps, w, args, tc_fp16, 0, 0, 0, status, st, dependent);
}

}  // namespace fm
