// Residual vector quantisation of few vectors: all layers of a stack in one kernel (sm_100a).  Same decisions as the chain of
// products and decision kernels in fm_rvq.cu (src/fast_mimi/model.py:2277-2291, :2408-2429).
//
// For few vectors that chain is bound by its launches: two a layer of 4 to 7 us each on the GPU and 4 us each on the host, for
// half a microsecond of products.  Here a thread-block cluster of 16 owns 16 or 32 vectors through the stack; block r has entries
// 128 r .. of every codebook.  Per layer
//   products   128 entries (FP16, 64 KB by TMA, two codebooks in flight) x the residuals, K = 256, on mma.sync: a tcgen05 tile would
//              be no faster for 32 columns and costs a hand-over through tensor memory
//   candidates entries within the vector's margin of the least approximate distance of the block's own: no fewer than those within
//              it of the least of all, and that one need not go round the cluster
//   decision   evaluated exactly in FP32, one warp each and four in flight, and the smallest (distance, index) over the cluster
//              wins: sent with st.async and counted where they arrive (a barrier of the cluster is a fence besides)
//   residual   every block subtracts the winner for itself: a warp holds its vectors in registers all along
// so a layer crosses the cluster once, and nothing but codes is written.  Stacks of 1 and 7 layers, in two rows of one grid, us: with two
// crossings behind barriers and 32 vectors a cluster -> here: 1 vector 44.7 -> 28.6, 16 47.8 -> 36.0, 63 49.3 -> 36.6, 112 56.1 -> 43.4, 150
// 57.9 -> 48.1, 224 58.2 -> 56.5; 1 and 31 layers of 63 vectors 212 -> 151.  (16 vectors a cluster: half the candidates and new
// residuals a block; 113 to 224 vectors need the clusters of 32.)
//
// The form with the stacks' input projections inside (512 -> 256 as split-precision products) saves two launches and the vectors' way
// through memory: 63 vectors, splitting + projection + search 47 us of kernels -> 38.7, 112 -> 82 us end to end with the convolution in front
// and the host's part.
#include "fm_common.cuh"
#include "fm_device_fact.h"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_rvq_key.h"
#include "fm_warp_mma.cuh"

namespace fm {

namespace rvqs {
constexpr int kCtas = 16, kEntries = 128;                      // of a cluster; of a block's share of a codebook
constexpr int kCodes = kCtas * kEntries;
constexpr int kDim = 256, kWarps = 16, kThreads = kWarps * 32;
constexpr int kHidden = 512, kProjected = kDim / kCtas;         // channels in front of the projection; dimensions of a block
constexpr int kBookBytes = kEntries * kDim * 2, kChunkBytes = kEntries * 128;
constexpr int kMaxLayers = 32;
constexpr int kMaxRows = 32;                                   // vectors of a cluster: 32 or 16
struct Shared {
  uint64_t full[2];
  uint64_t arrived[2];                             // all blocks' best candidates, of even and of odd layers
  uint64_t x_full;                                 // the projected vectors
  CtaCtl ctl;
  uint32_t pad;
  unsigned long long best[2][kMaxRows][kCtas];     // (distance, index) of every block's best candidate
  float min_in[8][kMaxRows];                       // of 16 entries of this block
  float margin[kMaxRows];
  unsigned long long best_in[2][kMaxRows];         // of this block's candidates
  int n_listed;
  uint16_t listed[kMaxRows * kEntries];            // candidates: vector * 128 + entry
};
constexpr int smem_bytes(int rows) { return 1024 + 2 * kBookBytes + rows * kDim * (2 + 4) + static_cast<int>(sizeof(Shared)); }

__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_async_f32(uint32_t addr, float v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_u64(uint32_t addr, unsigned long long v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar) : "memory");
}
}  // namespace rvqs

struct RvqStackArgs {
  struct Stack {
    const float* x;            // [rows, 256]
    const float* books;        // [layers, 2048, 256]
    const float* e_sq;         // [layers, 2048]
    long long* codes;          // [layers, rows]
    int layers;
    int w_row;                 // first row of the stack's projection in w_hi and w_lo
    float e_max[rvqs::kMaxLayers];
  };
  Stack stack[2];              // a row of the grid has one
  const float* frames;         // of the form with the projection inside: [rows, 512], which x is made from
  const uint16_t *w_hi, *w_lo; // [256 n_stacks, 512]
  int rows;
  float tau_rel;
};

template <int kRows, bool kProject>
__global__ void __launch_bounds__(rvqs::kThreads, 1)
rvq_stack_kernel(const __grid_constant__ CUtensorMap tmap_books0, const __grid_constant__ CUtensorMap tmap_books1,
                 const __grid_constant__ RvqStackArgs args, int* status) {
  using namespace rvqs;
  constexpr int kMine = kRows / kWarps;                        // vectors of a warp
  constexpr int kCols = kRows / 16;                            // columns of eight vectors of a warp's products
  const RvqStackArgs::Stack& a = args.stack[blockIdx.y];
  const CUtensorMap* tmap_books = blockIdx.y == 0 ? &tmap_books0 : &tmap_books1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_book = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_x = smem_book + 2 * kBookBytes;                // FP16 residuals: four chunks of 64 dimensions
  float* exact_x = reinterpret_cast<float*>(smem_x + kRows * kDim * 2);      // the residuals in FP32, for whichever warp needs them
  Shared* sh = reinterpret_cast<Shared*>(exact_x + kRows * kDim);
  CtaCtl* ctl = &sh->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = static_cast<int>(threadIdx.x);
  const int rank = static_cast<int>(cluster_cta_rank());
  const int r0 = static_cast<int>(blockIdx.x) / kCtas * kRows;
  const int n = args.rows - r0 < kRows ? args.rows - r0 : kRows;
  // read early: a status set before this call leaves the stores out
  const bool skip = status != nullptr && *reinterpret_cast<volatile int*>(status) != 0;
  auto load_book = [&](int l) {
    uint8_t* dst = smem_book + (l & 1) * kBookBytes;
    mbar_arrive_expect_tx(&sh->full[l & 1], kBookBytes);
#pragma unroll
    for (int kc = 0; kc < kDim / 64; ++kc) tma_load_2d(dst + kc * kChunkBytes, tmap_books, &sh->full[l & 1], kc * 64, l * kCodes + rank * kEntries);
  };
  if (tid == 0) {
    mbar_init(&sh->full[0], 1);
    mbar_init(&sh->full[1], 1);
    mbar_init(&sh->arrived[0], 1);
    mbar_init(&sh->arrived[1], 1);
    ctl->abort = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&sh->arrived[0], kRows * kCtas * 8);
    mbar_arrive_expect_tx(&sh->arrived[1], kRows * kCtas * 8);
    if (kProject) {
      mbar_init(&sh->x_full, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&sh->x_full, kRows * kDim * 4);
    }
    load_book(0);
    if (!kProject && a.layers > 1) load_book(1);
  }

  // This warp's vectors, eight values a lane, in every block of the cluster.
  float x[kMine][8];
  if constexpr (kProject) {
    // Projection: 16 of the 256 dimensions a block, 32 of the 512 channels a warp.  Operands are FP16 hi + lo parts (of the frames: made
    // here), the small terms in a sum of their own; K is permuted alike in both, so that a lane's share of 32 channels of a row lies
    // together.
    __syncthreads();
    cluster_arrive_relaxed();                                  // this block runs: its shared memory may be written
    const int g = lane >> 2, q = lane & 3;
    float* red = reinterpret_cast<float*>(smem_book + kBookBytes);
    uint4 w[2][2];                                             // rows g and g + 8; hi and lo
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const size_t at = static_cast<size_t>(a.w_row + rank * kProjected + e * 8 + g) * kHidden + warp * 32 + q * 8;
      w[e][0] = __ldg(reinterpret_cast<const uint4*>(args.w_hi + at));
      w[e][1] = __ldg(reinterpret_cast<const uint4*>(args.w_lo + at));
    }
    float4 v[kRows / 8][2];
#pragma unroll
    for (int t = 0; t < kRows / 8; ++t) {
      const int f = t * 8 + g;
      const float4* p = reinterpret_cast<const float4*>(args.frames + static_cast<size_t>(r0 + (f < n ? f : 0)) * kHidden + warp * 32 + q * 8);
      v[t][0] = __ldg(p);
      v[t][1] = __ldg(p + 1);
    }
#pragma unroll
    for (int t = 0; t < kRows / 8; ++t) {
      uint4 hi, lo;
      split_half8(v[t][0], v[t][1], hi, lo);
      float small[4] = {0.f, 0.f, 0.f, 0.f}, main[4] = {0.f, 0.f, 0.f, 0.f};
      mma_16x8x32<__half>(small, w[0][0], w[1][0], lo);
      mma_16x8x32<__half>(small, w[0][1], w[1][1], hi);
      mma_16x8x32<__half>(main, w[0][0], w[1][0], hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int f = t * 8 + 2 * q + (e & 1), o = g + 8 * (e >> 1);
        red[(warp * kRows + f) * kProjected + (o ^ ((q & 1) << 3))] = small[e] + main[e];
      }
    }
    __syncthreads();
    cluster_wait();
    for (int i = tid; i < kRows * kProjected; i += kThreads) {
      const int f = i / kProjected, o = i % kProjected;
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) sum += red[(k * kRows + f) * kProjected + (o ^ (((f >> 1) & 1) << 3))];
      if (f >= n) sum = 0.f;
      const uint32_t at = smem_u32(exact_x + f * kDim + rank * kProjected + o), bar = smem_u32(&sh->x_full);
#pragma unroll
      for (uint32_t peer = 0; peer < kCtas; ++peer) st_async_f32(map_to_cta(at, peer), sum, map_to_cta(bar, peer));
    }
    if (a.layers > 1) {                                        // the second codebook comes where the partial sums were
      fence_proxy_async_smem();
      __syncthreads();
      if (tid == 0) load_book(1);
    }
    mbar_wait_cluster(&sh->x_full, 0, ctl, status, kErrWaitConsumer);
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < kMine; ++i) {
    const int f = warp + kWarps * i;
#pragma unroll
    for (int k = 0; k < 8; ++k) x[i][k] = 0.f;
    if (f < n) {
      const float4* p = reinterpret_cast<const float4*>(kProject ? exact_x + f * kDim + lane * 8 : a.x + static_cast<size_t>(r0 + f) * kDim + lane * 8);
      const float4 u = kProject ? p[0] : __ldcg(p), v = kProject ? p[1] : __ldcg(p + 1);
      x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w; x[i][4] = v.x; x[i][5] = v.y; x[i][6] = v.z; x[i][7] = v.w;
    }
  }
  // FP16 copy, margin (the same sums in the same order as in fm_rvq.cu) and an empty set of candidates for the layer to come
  auto open_layer = [&](int l) {
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int f = warp + kWarps * i;
      float xx = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) xx = fmaf(x[i][k], x[i][k], xx);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) xx += __shfl_xor_sync(0xffffffffu, xx, o);
      *reinterpret_cast<uint4*>(smem_x + (lane >> 3) * (kRows * 128) + sw128_offset(f, lane & 7)) =
          make_uint4(Pack16<__half>::pack(x[i][0], x[i][1]), Pack16<__half>::pack(x[i][2], x[i][3]),
                     Pack16<__half>::pack(x[i][4], x[i][5]), Pack16<__half>::pack(x[i][6], x[i][7]));
      float4* exact = reinterpret_cast<float4*>(exact_x + f * kDim + lane * 8);
      exact[0] = make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
      exact[1] = make_float4(x[i][4], x[i][5], x[i][6], x[i][7]);
      if (lane == 0) {
        sh->margin[f] = rvq_margin(xx, a.e_max[l], args.tau_rel);
        sh->best_in[l & 1][f] = kRvqNoKey;
      }
    }
    if (tid == 0) sh->n_listed = 0;
  };
  open_layer(0);
  __syncthreads();
  if (!kProject) cluster_arrive_relaxed();                     // this block runs: its shared memory may be written

  const int g = lane >> 2, cpair = (lane & 3) * 2;
  const int mt = warp >> 1, nh = warp & 1;                     // 16 entries x half of the vectors of the products
  const int f0 = nh * (kRows / 2) + cpair;
  for (int l = 0; l < a.layers; ++l) {
    const float* sq = a.e_sq + static_cast<size_t>(l) * kCodes + rank * kEntries + mt * 16 + g;
    const float e_sq[2] = {__ldg(sq), __ldg(sq + 8)};
    mbar_wait(&sh->full[l & 1], static_cast<uint32_t>(l >> 1) & 1u, ctl, status, kErrWaitTma);
    float d[kCols][4];
#pragma unroll
    for (int nt = 0; nt < kCols; ++nt) d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.f;
    {
      const uint32_t book = smem_u32(smem_book + (l & 1) * kBookBytes), vec = smem_u32(smem_x);
#pragma unroll
      for (int kc = 0; kc < kDim / 64; ++kc) {
#pragma unroll
        for (int ks = 0; ks < 4; ks += 2) {
          uint32_t ea[2][4], xb[kCols][4];
#pragma unroll
          for (int s = 0; s < 2; ++s) ldmatrix4(ea[s], book + kc * kChunkBytes + sw128_offset(mt * 16 + (lane & 15), 2 * (ks + s) + (lane >> 4)));
#pragma unroll
          for (int nt = 0; nt < kCols; ++nt)
            ldmatrix4(xb[nt], vec + kc * (kRows * 128) + sw128_offset(nh * (kRows / 2) + nt * 8 + (lane & 7), 2 * ks + (lane >> 3)));
#pragma unroll
          for (int s = 0; s < 2; ++s) {
#pragma unroll
            for (int nt = 0; nt < kCols; ++nt) mma_16x8x16<__half>(d[nt], ea[s], xb[nt][2 * s], xb[nt][2 * s + 1]);
          }
        }
      }
    }
    // approximate distances: entries g and g + 8 of the tile, vectors cpair and cpair + 1 of each eight
#pragma unroll
    for (int nt = 0; nt < kCols; ++nt) {
      float m[2];
#pragma unroll
      for (int e = 0; e < 4; ++e) d[nt][e] = fmaf(-2.f, d[nt][e], e_sq[e >> 1]);
      m[0] = fminf(d[nt][0], d[nt][2]);
      m[1] = fminf(d[nt][1], d[nt][3]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        m[0] = fminf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
        m[1] = fminf(m[1], __shfl_xor_sync(0xffffffffu, m[1], o));
      }
      if (g == 0) *reinterpret_cast<float2*>(&sh->min_in[mt][f0 + nt * 8]) = make_float2(m[0], m[1]);
    }
    __syncthreads();
    if (tid == 0 && l + 2 < a.layers) load_book(l + 2);        // the products are done with this layer's codebook
    // Candidates: within the margin of the least of this block's own entries, which all that are within it of the least of all are.
#pragma unroll
    for (int nt = 0; nt < kCols; ++nt) {
      float2 m = *reinterpret_cast<const float2*>(&sh->min_in[0][f0 + nt * 8]);
#pragma unroll
      for (int i = 1; i < 8; ++i) {
        const float2 o = *reinterpret_cast<const float2*>(&sh->min_in[i][f0 + nt * 8]);
        m.x = fminf(m.x, o.x);
        m.y = fminf(m.y, o.y);
      }
      const float2 margin = *reinterpret_cast<const float2*>(&sh->margin[f0 + nt * 8]);
      const float limit[2] = {m.x + margin.x, m.y + margin.y};
      if (warp == nh && g == 0) {                              // one that is not finite: no candidate in any block, whatever the others find
        if (!(limit[0] == limit[0])) atomicMin(&sh->best_in[l & 1][f0 + nt * 8], kRvqNoCandidate);
        if (!(limit[1] == limit[1])) atomicMin(&sh->best_in[l & 1][f0 + nt * 8 + 1], kRvqNoCandidate);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int f = f0 + nt * 8 + (e & 1), j = mt * 16 + g + 8 * (e >> 1);
        if (f < n && d[nt][e] <= limit[e & 1]) sh->listed[atomicAdd(&sh->n_listed, 1)] = static_cast<uint16_t>(f * kEntries + j);
      }
    }
    __syncthreads();
    // ---- exactly, a warp up to four at a time; the smaller distance wins, on ties the lower index (argmin's rule)
    const int n_listed = sh->n_listed;
    for (int c0 = warp; c0 < n_listed; c0 += 4 * kWarps) {
      float4 u[4], v[4];
      int at[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        at[i] = sh->listed[c0 + i * kWarps < n_listed ? c0 + i * kWarps : c0];
        const float4* er = reinterpret_cast<const float4*>(a.books + (static_cast<size_t>(l) * kCodes + rank * kEntries + at[i] % kEntries) * kDim + lane * 8);
        u[i] = __ldg(er);
        v[i] = __ldg(er + 1);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int f = at[i] / kEntries, j = rank * kEntries + at[i] % kEntries;
        const float4* xr = reinterpret_cast<const float4*>(exact_x + f * kDim + lane * 8);
        const float4 xa = xr[0], xb = xr[1];
        const float ev[8] = {u[i].x, u[i].y, u[i].z, u[i].w, v[i].x, v[i].y, v[i].z, v[i].w}, xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float t = xv[k] - ev[k];
          acc = fmaf(t, t, acc);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        // a distance that is not finite loses to every other and leaves index 0, as where nothing is smaller than the best so far
        const unsigned long long key = acc < INFINITY ? (static_cast<unsigned long long>(__float_as_uint(acc)) << 32) | static_cast<unsigned>(j)
                                                      : kRvqNotFinite;
        if (lane == 0 && c0 + i * kWarps < n_listed) atomicMin(&sh->best_in[l & 1][f], key);
      }
    }
    __syncthreads();
    if (!kProject && l == 0) cluster_wait();
    if (tid < kRows * kCtas) {                                 // one of the block's best to one of 16 blocks, counted where it arrives
      const int f = tid % kRows;
      const uint32_t peer = static_cast<uint32_t>(tid / kRows);
      st_async_u64(map_to_cta(smem_u32(&sh->best[l & 1][f][rank]), peer), sh->best_in[l & 1][f], map_to_cta(smem_u32(&sh->arrived[l & 1]), peer));
    }
    const bool whole = mbar_wait_cluster(&sh->arrived[l & 1], static_cast<uint32_t>(l >> 1) & 1u, ctl, status, kErrWaitConsumer);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int f = warp + kWarps * i;
      unsigned long long best = sh->best[l & 1][f][lane & 15];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other < best ? other : best;
      }
      const int entry = rvq_entry_of(best, kCodes), j = entry < 0 ? 0 : entry;
      const bool none = entry < 0;                             // a residual that is not finite
      if (rank == 0 && lane == 0 && f < n && !skip && whole) {       // (after a wait that gave up: words of no meaning)
        a.codes[static_cast<size_t>(l) * args.rows + r0 + f] = j;
        if (none && status != nullptr) atomicMax(status, static_cast<int>(kErrNonFinite));
      }
      if (l + 1 < a.layers) {
        const float4* er = reinterpret_cast<const float4*>(a.books + (static_cast<size_t>(l) * kCodes + j) * kDim + lane * 8);
        const float4 u = __ldg(er), v = __ldg(er + 1);
        x[i][0] -= u.x; x[i][1] -= u.y; x[i][2] -= u.z; x[i][3] -= u.w;
        x[i][4] -= v.x; x[i][5] -= v.y; x[i][6] -= v.z; x[i][7] -= v.w;
      }
    }
    if (l + 1 < a.layers) {
      if (tid == 0) mbar_arrive_expect_tx(&sh->arrived[l & 1], kRows * kCtas * 8);       // for the layer after that
      open_layer(l + 1);
      __syncthreads();
    }
  }
  if (ctl->abort) __nanosleep(20000);
  cluster_sync_all();                                          // nobody still writes into a block that has left
}

namespace {
// Clusters of 16 blocks that the device runs at once (0: none, or not to be found out just now).
int stack_slots() {
  static DeviceFact slots;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const int n = slots.get(dev, [] {
    const auto allow = [](auto kern, int bytes) {
      return ensure_dynamic_smem(reinterpret_cast<const void*>(kern), bytes) == 0 &&
             cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    };
    if (!allow(rvq_stack_kernel<16, false>, rvqs::smem_bytes(16)) || !allow(rvq_stack_kernel<32, false>, rvqs::smem_bytes(32)) ||
        !allow(rvq_stack_kernel<16, true>, rvqs::smem_bytes(16)) || !allow(rvq_stack_kernel<32, true>, rvqs::smem_bytes(32))) {
      (void)cudaGetLastError();
      return -1;
    }
    return resident_clusters(rvq_stack_kernel<32, false>, rvqs::kThreads, rvqs::smem_bytes(32), rvqs::kCtas);
  });
  return n > 0 ? n : 0;
}
}  // namespace

// As many vectors as the device's clusters hold at once (7 x 32 on a B200): a second wave costs as much as the first, the chain
// next to nothing more (7 layers of 224 vectors 55 us here, 72 there; 225 vectors 99 and 70).
// Two stacks are two rows of one grid, whether or not the device holds both at once.
bool rvq_stack_takes(const RvqStack* stacks, int n_stacks, long long rows, int n_codes) {
  for (int i = 0; i < n_stacks; ++i)
    if (stacks[i].layers > rvqs::kMaxLayers) return false;
  return n_codes == rvqs::kCodes && rows <= static_cast<long long>(rvqs::kMaxRows) * stack_slots();
}

int launch_rvq_stack(const RvqStack* stacks, int n_stacks, long long rows, float tau_rel, int* status, cudaStream_t st, const RvqFrames* from) {
  using namespace rvqs;
  if (n_stacks < 1 || n_stacks > 2 || !(tau_rel >= 0.f)) return -1;
  if (from != nullptr && (reinterpret_cast<uintptr_t>(from->x) | reinterpret_cast<uintptr_t>(from->w_hi) | reinterpret_cast<uintptr_t>(from->w_lo)) & 15u) return -3;
  RvqStackArgs a = {};
  CUtensorMap maps[2];
  const int longer = n_stacks == 2 && stacks[1].layers > stacks[0].layers ? 1 : 0;     // comes first
  for (int i = 0; i < n_stacks; ++i) {
    const RvqStack& s = stacks[i == 0 ? longer : 1 - longer];
    if ((s.residual == nullptr && from == nullptr) || s.books16 == nullptr || s.books == nullptr || s.e_sq == nullptr || s.codes == nullptr) return -1;
    if ((reinterpret_cast<uintptr_t>(s.residual) | reinterpret_cast<uintptr_t>(s.books) | reinterpret_cast<uintptr_t>(s.books16)) & 15u) return -3;
    RvqStackArgs::Stack& d = a.stack[i];
    d.x = s.residual;
    d.books = s.books;
    d.e_sq = s.e_sq;
    d.codes = s.codes;
    d.layers = s.layers;
    d.w_row = (i == 0 ? longer : 1 - longer) * kDim;
    for (int l = 0; l < s.layers; ++l) {
      if (!(s.e_max[l] >= 0.f)) return -1;
      d.e_max[l] = s.e_max[l];
    }
    const int rc = encode_rows_16bit(&maps[i], s.books16, static_cast<uint64_t>(s.layers) * kCodes, kDim, kEntries, 64);
    if (rc != 0) return rc;
  }
  if (n_stacks == 1) maps[1] = maps[0];
  a.rows = static_cast<int>(rows);
  a.tau_rel = tau_rel;
  // 16 vectors a cluster while the device holds all clusters of the longer stack at once and the other one's, if some of those have to
  // wait, end no later.
  const int few = static_cast<int>((rows + 15) / 16), slots = stack_slots();
  const bool sixteen = few <= slots && (n_stacks == 1 || 2 * few <= slots || 2 * a.stack[1].layers <= a.stack[0].layers);
  const int per = sixteen ? 16 : 32;
  if (from != nullptr) {
    a.frames = from->x;
    a.w_hi = static_cast<const uint16_t*>(from->w_hi);
    a.w_lo = static_cast<const uint16_t*>(from->w_lo);
  }
  auto kern = from != nullptr ? (sixteen ? rvq_stack_kernel<16, true> : rvq_stack_kernel<32, true>)
                              : (sixteen ? rvq_stack_kernel<16, false> : rvq_stack_kernel<32, false>);
  return launch_kernel(kern, dim3(static_cast<unsigned>((rows + per - 1) / per) * kCtas, static_cast<unsigned>(n_stacks)), kThreads, smem_bytes(per), st, kCtas,
                       0, maps[0], maps[1], a, status);
}

}  // namespace fm
