// LayerNorm and the product behind it in one kernel, for few rows (sm_100a):  q | k | v with RoPE, or gelu(.),  of
// LayerNorm(x) W^T with 512 channels.  Reference: src/fast_mimi/model.py:2021-2024 with :1897-1912 and :1990-1999.
//
// Latency-bound: at one clip's rows a LayerNorm launch (1.5 us of memory round trip and reductions) and the product
// behind it (2.5 us) each pay a kernel boundary.  Here a block owns `kRows` rows (16 or 32) x 64 outputs (one head):
// its eight epilogue warps normalise the rows, one warp per row at a time, straight into the swizzled operand tile, and
// the whole K = 512 of its weight slice (64 KB) sits in shared memory, requested before the wait for the kernel in front.
// There is no K split, hence no cluster and no reduction.  Every block repeats the normalisation of its rows (32 or 64 KB
// of x from L2), which is what limits the rows.
//
// The tensor core multiplies 128 rows whatever kRows is; the operand tile of a K chunk is only kRows rows high, so what
// it reads past them is the next chunk (or the weights): finite or not, those products stay in accumulator rows that
// nobody reads.
//
// Warps 0-7: LayerNorm, then accumulator and epilogue.  Warp 8: weights.  Warp 9: MMA.
#include "fm_launch.h"
#include "fm_small_tile.cuh"

namespace fm {

namespace lnlin {
constexpr int kHidden = 512;
constexpr int kBlockN = 64;
constexpr int kChunks = kHidden / 64;
constexpr int kWBytes = kBlockN * 128;          // one K chunk of the weight slice
constexpr int kWarps = 8;
constexpr int kThreads = (kWarps + 2) * 32;
constexpr int kTmemCols = 64;
struct Barriers {
  uint64_t w_full[2];                           // the two halves of the weight slice
  uint64_t acc_full;
  uint32_t tmem_base;
  CtaCtl ctl;
};
// The operand tile comes first: the tensor core reads up to 128 - kRows rows past its last chunk, i.e. into the weights.
constexpr int smem_bytes(int rows) { return 1024 + kChunks * (rows * 128 + kWBytes) + rows * 256 + 64; }
static_assert(sizeof(Barriers) <= 64, "barrier block too large");
}  // namespace lnlin

struct LnArgs {
  const void* x;          // [M, 512]
  ParamVec weight;
  ParamVec bias;
  float eps;
  int opens_chain;        // first kernel of a chain: lets the next one start only after its own wait
};

// kIn: type of x (0 BF16, 1 FP16, 2 FP32); kTc: type of the product's operands (0 BF16, 1 FP16); kOut: kTc, or 3 = q | k | v
template <int kIn, int kTc, int kOut, typename VT, int kRows>
__global__ void __launch_bounds__(lnlin::kThreads)
ln_linear_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ LnArgs ln,
                 const __grid_constant__ SmallArgs args, uint32_t idesc, int* status) {
  using namespace lnlin;
  using TOp = typename std::conditional<kTc == 1, __half, __nv_bfloat16>::type;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_h = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_w = smem_h + kChunks * kRows * 128;
  uint8_t* smem_o = smem_w + kChunks * kWBytes;
  Barriers* bars = reinterpret_cast<Barriers*>(smem_o + kRows * 256);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntile = static_cast<int>(blockIdx.x);
  const int m0 = static_cast<int>(blockIdx.y) * kRows;
  // read early: a status set before this chain began stops every kernel of it (the stores are left out)
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  if (threadIdx.x == 0) {
    mbar_init(&bars->w_full[0], 1);
    mbar_init(&bars->w_full[1], 1);
    mbar_init(&bars->acc_full, 1);
    bars->ctl.abort = 0;
    fence_mbar_init();
  }
  if (warp == kWarps + 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  CtaCtl* ctl = &bars->ctl;

  if (warp == kWarps && lane == 0) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      mbar_arrive_expect_tx(&bars->w_full[half], kChunks / 2 * kWBytes);
#pragma unroll
      for (int kc = half * kChunks / 2; kc < (half + 1) * kChunks / 2; ++kc)
        tma_load_2d(smem_w + kc * kWBytes, &tmap_w, &bars->w_full[half], kc * 64, ntile * kBlockN);
    }
  }
  if (!ln.opens_chain) griddep_launch();
  PieceOperands ops;
  const int n_rows = args.M - m0 < kRows ? args.M - m0 : kRows;
  const int n_items = skip ? 0 : n_rows * 8;
  int item = static_cast<int>(threadIdx.x);
  if (warp < kWarps) {
    // this lane's channels: 4 * lane + 128 * j + (0..3)
    uint4 w_raw[4], b_raw[4];
    griddep_wait();
    if (ln.opens_chain) griddep_launch();
    float v[kRows / kWarps][4][4];
#pragma unroll
    for (int i = 0; i < kRows / kWarps; ++i) {
      const int r = i * kWarps + warp;
      if (r < n_rows) {
#pragma unroll
        for (int j = 0; j < 4; ++j) load4<kIn>(ln.x, static_cast<long long>(m0 + r) * kHidden + 128 * j + 4 * lane, v[i][j]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j][0] = v[i][j][1] = v[i][j][2] = v[i][j][3] = 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w_raw[j] = ln.weight.raw4<kIn == 2>(128 * j + 4 * lane);
      b_raw[j] = ln.bias.raw4<kIn == 2>(128 * j + 4 * lane);
    }
    if (item < n_items) load_operands<kOut>(args, m0 + (item >> 3), ntile, item & 7, ops);
    // the same sums in the same order as layernorm512_kernel
    float sum[kRows / kWarps], sq[kRows / kWarps];
#pragma unroll
    for (int i = 0; i < kRows / kWarps; ++i) {
      sum[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i] += (v[i][j][0] + v[i][j][1]) + (v[i][j][2] + v[i][j][3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < kRows / kWarps; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
    }
#pragma unroll
    for (int i = 0; i < kRows / kWarps; ++i) {
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
      for (int i = 0; i < kRows / kWarps; ++i) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
    }
    float w[4][4], b[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 wf = ln.weight.value4<kIn == 2>(w_raw[j]);
      const float4 bf = ln.bias.value4<kIn == 2>(b_raw[j]);
      w[j][0] = wf.x; w[j][1] = wf.y; w[j][2] = wf.z; w[j][3] = wf.w;
      b[j][0] = bf.x; b[j][1] = bf.y; b[j][2] = bf.z; b[j][3] = bf.w;
    }
#pragma unroll
    for (int i = 0; i < kRows / kWarps; ++i) {
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
  __syncthreads();                          // the operand tile is complete
  if (warp == kWarps + 1) {
    const bool one = elect_one();
    tc_fence_after_sync();
    const uint64_t a_desc = umma_desc_sw128(smem_u32(smem_h)), b_desc = umma_desc_sw128(smem_u32(smem_w));
    for (int kc = 0; kc < kChunks; ++kc) {
      if (kc % (kChunks / 2) == 0) {
        mbar_wait(&bars->w_full[kc / (kChunks / 2)], 0, ctl, status, kErrWaitTma);
        tc_fence_after_sync();
      }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        if (one)
          tc_mma_ss(tmem_base, a_desc + static_cast<uint64_t>(kc * kRows * 128 >> 4) + 2u * ks,
                    b_desc + static_cast<uint64_t>(kc * kWBytes >> 4) + 2u * ks, idesc, (kc | ks) != 0 ? 1u : 0u);
    }
    if (one) tc_commit(&bars->acc_full);
    __syncwarp();
  }
  if (warp == 0) {
    // rows 0 .. kRows - 1 sit in the first 32 lanes of tensor memory
    mbar_wait(&bars->acc_full, 0, ctl, status, kErrWaitMma);
    tc_fence_after_sync();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t a[32];
      tmem_ld32(tmem_base + h * 32, a);
      tmem_ld_wait();
      if (lane < kRows) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(smem_o + small::red_offset(lane, h * 8 + c, lane)) =
              make_uint4(a[4 * c], a[4 * c + 1], a[4 * c + 2], a[4 * c + 3]);
      }
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp < kWarps && item < n_items) {    // kRows * 8 pieces, one per thread at most
    const int local = item >> 3, j = item & 7;
    const float4 a = *reinterpret_cast<const float4*>(smem_o + small::red_offset(local, j, local));
    const float4 c = *reinterpret_cast<const float4*>(smem_o + small::red_offset(local, j + 8, local));
    float lo[4] = {a.x, a.y, a.z, a.w}, hi[4] = {c.x, c.y, c.z, c.w};
    finish_piece<kOut, VT>(args, lo, hi, ops, m0 + local, ntile, j, status);
  }
  if (ctl->abort) __nanosleep(20000);
  if (warp == kWarps + 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

static long long blocks_for(int M, int N, int rows) { return static_cast<long long>((M + rows - 1) / rows) * (N / lnlin::kBlockN); }
// 16 rows per block while that is at most one block per SM, else 32; beyond one block per SM of those the separate
// LayerNorm kernel is cheaper.  More blocks than SMs do not pay: two of them leave no room on an SM for the next kernel's
// block, which then starts (and asks for its weights) only when they have ended (125 rows: fc2 began 5 us after fc1's
// first blocks were done instead of 2).
static int rows_per_block(int M, int N) { return blocks_for(M, N, 16) <= sm_count() ? 16 : 32; }

bool few_rows_with_norm(int M, int N) { return blocks_for(M, N, 32) <= sm_count(); }

template <int kIn, int kTc, int kOut, typename VT>
static int launch_rows(const CUtensorMap& tmap_w, const LnArgs& ln, const SmallArgs& args, uint32_t idesc, int* status,
                       cudaStream_t st, int dependent) {
  using namespace lnlin;
  const int rows = rows_per_block(args.M, args.N);
  auto kern = rows == 16 ? ln_linear_kernel<kIn, kTc, kOut, VT, 16> : ln_linear_kernel<kIn, kTc, kOut, VT, 32>;
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem_bytes(rows));
  if (rc != 0) return rc;
  return launch_kernel(kern, dim3(args.N / kBlockN, (args.M + rows - 1) / rows), kThreads, smem_bytes(rows), st, 1, dependent,
                       tmap_w, ln, args, idesc, status);
}

template <int kIn, int kTc>
static int launch_typed(const CUtensorMap& tmap_w, const LnArgs& ln, const SmallArgs& args, uint32_t idesc, int qkv, int value_fp16,
                        int* status, cudaStream_t st, int dependent) {
  if (!qkv) return launch_rows<kIn, kTc, kTc, __half>(tmap_w, ln, args, idesc, status, st, dependent);
  if (value_fp16) return launch_rows<kIn, kTc, 3, __half>(tmap_w, ln, args, idesc, status, st, dependent);
  return launch_rows<kIn, kTc, 3, __nv_bfloat16>(tmap_w, ln, args, idesc, status, st, dependent);
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
  const LnArgs ln = {x, weight, bias, eps, opens_chain};
  const int fmt = tc_fp16 ? 0 : 1;
  const uint32_t idesc = umma_idesc_f16(128, lnlin::kBlockN, fmt, fmt, 0, 0);
  using Fn = int (*)(const CUtensorMap&, const LnArgs&, const SmallArgs&, uint32_t, int, int, int*, cudaStream_t, int);
  static const Fn table[3][2] = {{launch_typed<0, 0>, launch_typed<0, 1>}, {launch_typed<1, 0>, launch_typed<1, 1>},
                                 {launch_typed<2, 0>, launch_typed<2, 1>}};
  return table[x_dtype][tc_fp16 ? 1 : 0](tmap_w, ln, args, idesc, qkv, value_fp16, status, st, dependent);
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
