// Residual vector quantisation of few vectors: all layers of a stack in one kernel (sm_100a).  Same decisions as the chain of
// products and decision kernels in fm_rvq.cu (src/fast_mimi/model.py:2277-2291, :2408-2429).
//
// For few vectors that chain is bound by its launches: two a layer of 4 to 7 us each on the GPU and 4 us each on the host, for
// half a microsecond of products.  Here a thread-block cluster of 16 owns 32 vectors through the stack; block r has entries
// 128 r .. of every codebook.  Per layer
//   products   128 entries (FP16, 64 KB by TMA, two codebooks in flight) x 32 residuals, K = 256, on mma.sync: a tcgen05 tile would
//              be no faster for 32 columns and costs a hand-over through tensor memory
//   minimum    of the approximate distances: in the block, then over the cluster through distributed shared memory
//   decision   entries within the vector's margin of it are evaluated exactly in FP32, one warp each, and the smallest
//              (distance, index) over the cluster wins
//   residual   every block subtracts the winner for itself: a warp holds its two vectors in registers all along
// so a layer crosses the cluster twice, and nothing but codes is written.  63 vectors: 7 layers 66 -> 55 us, 31 layers 273 -> 219
// us, and 16 launches less for stacks of 1 and 7 layers, 18 otherwise (a 5 s utterance end to end, bound by the host, 200 -> 183 us;
// both stacks as two rows of one grid, which the device runs side by side up to three clusters each, 176 -> 172, no more than runs differ by).  Of the 12300 cycles of a layer the
// two crossings take 4500, the products 2100 (ldmatrix at the rate of shared memory), the exact distances 1400, the new residual 2700.
#include "fm_common.cuh"
#include "fm_device_fact.h"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_warp_mma.cuh"

namespace fm {

namespace rvqs {
constexpr int kCtas = 16, kRows = 32, kEntries = 128;          // of a cluster; of a block's share of a codebook
constexpr int kCodes = kCtas * kEntries;
constexpr int kDim = 256, kWarps = 16, kThreads = kWarps * 32;
constexpr int kBookBytes = kEntries * kDim * 2, kChunkBytes = kEntries * 128;
constexpr int kMaxLayers = 32;
struct Shared {
  uint64_t full[2];
  CtaCtl ctl;
  uint32_t pad[3];
  unsigned long long best[kRows][kCtas];     // (distance, index) of every block's best candidate
  float min_of[kRows][kCtas];                // every block's smallest approximate distance
  float min_in[8][kRows];                    // of 16 entries of this block
  float limit[kRows];
  float margin[kRows];
  unsigned long long best_in[kRows];         // of this block's candidates
  int n_listed;
  uint16_t listed[kRows * kEntries];         // candidates: vector * 128 + entry
};
constexpr int kSmemBytes = 1024 + 2 * kBookBytes + kRows * kDim * (2 + 4) + static_cast<int>(sizeof(Shared));

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
}  // namespace rvqs

struct RvqStackArgs {
  struct Stack {
    const float* x;            // [rows, 256]
    const float* books;        // [layers, 2048, 256]
    const float* e_sq;         // [layers, 2048]
    long long* codes;          // [layers, rows]
    int layers;
    float e_max[rvqs::kMaxLayers];
  };
  Stack stack[2];              // a row of the grid has one
  int rows;
  float tau_rel;
};

__global__ void __launch_bounds__(rvqs::kThreads, 1)
rvq_stack_kernel(const __grid_constant__ CUtensorMap tmap_books0, const __grid_constant__ CUtensorMap tmap_books1,
                 const __grid_constant__ RvqStackArgs args, int* status) {
  using namespace rvqs;
  const RvqStackArgs::Stack& a = args.stack[blockIdx.y];
  const CUtensorMap* tmap_books = blockIdx.y == 0 ? &tmap_books0 : &tmap_books1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_book = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_x = smem_book + 2 * kBookBytes;                // FP16 residuals: four chunks of 64 dimensions, 32 rows each
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
    ctl->abort = 0;
    fence_mbar_init();
    load_book(0);
    if (a.layers > 1) load_book(1);
  }

  // This warp's two vectors, eight values a lane, in every block of the cluster.
  float x[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int f = warp + kWarps * i;
#pragma unroll
    for (int k = 0; k < 8; ++k) x[i][k] = 0.f;
    if (f < n) {
      const float4* p = reinterpret_cast<const float4*>(a.x + static_cast<size_t>(r0 + f) * kDim + lane * 8);
      const float4 u = __ldcg(p), v = __ldcg(p + 1);
      x[i][0] = u.x; x[i][1] = u.y; x[i][2] = u.z; x[i][3] = u.w; x[i][4] = v.x; x[i][5] = v.y; x[i][6] = v.z; x[i][7] = v.w;
    }
  }
  // FP16 copy, margin (the same sums in the same order as in fm_rvq.cu) and an empty set of candidates for the layer to come
  auto open_layer = [&](int l) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
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
        sh->best_in[f] = ~0ull;
      }
    }
    if (tid == 0) sh->n_listed = 0;
  };
  open_layer(0);
  __syncthreads();
  cluster_arrive();                                            // this block runs: its shared memory may be written

  const int g = lane >> 2, cpair = (lane & 3) * 2;
  const int mt = warp >> 1, nh = warp & 1;                     // 16 entries x 16 vectors of the products
  for (int l = 0; l < a.layers; ++l) {
    const float* sq = a.e_sq + static_cast<size_t>(l) * kCodes + rank * kEntries + mt * 16 + g;
    const float e_sq[2] = {__ldg(sq), __ldg(sq + 8)};
    mbar_wait(&sh->full[l & 1], static_cast<uint32_t>(l >> 1) & 1u, ctl, status, kErrWaitTma);
    float d[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.f;
    {
      const uint32_t book = smem_u32(smem_book + (l & 1) * kBookBytes), vec = smem_u32(smem_x);
#pragma unroll
      for (int kc = 0; kc < kDim / 64; ++kc) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          uint32_t ea[4], xb[4];
          ldmatrix4(ea, book + kc * kChunkBytes + sw128_offset(mt * 16 + (lane & 15), 2 * ks + (lane >> 4)));
          ldmatrix4(xb, vec + kc * (kRows * 128) + sw128_offset(nh * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * ks + ((lane >> 3) & 1)));
          mma_16x8x16<__half>(d[0], ea, xb[0], xb[1]);
          mma_16x8x16<__half>(d[1], ea, xb[2], xb[3]);
        }
      }
    }
    // approximate distances: entries g and g + 8 of the tile, vectors cpair and cpair + 1 of each eight
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
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
      if (g == 0) *reinterpret_cast<float2*>(&sh->min_in[mt][nh * 16 + nt * 8 + cpair]) = make_float2(m[0], m[1]);
    }
    __syncthreads();
    if (tid == 0 && l + 2 < a.layers) load_book(l + 2);        // the products are done with this layer's codebook
    if (l == 0) cluster_wait();
    {
      const int f = tid & 31, peer = tid >> 5;                 // one of the block's 32 minima to one of 16 blocks
      float m = sh->min_in[0][f];
#pragma unroll
      for (int i = 1; i < 8; ++i) m = fminf(m, sh->min_in[i][f]);
      st_cluster_f32(map_to_cta(smem_u32(&sh->min_of[f][rank]), static_cast<uint32_t>(peer)), m);
    }
    cluster_sync_all();
    {
      const int f = tid >> 4;
      float m = sh->min_of[f][tid & 15];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((tid & 15) == 0) sh->limit[f] = m + sh->margin[f];
    }
    __syncthreads();
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int f = nh * 16 + nt * 8 + cpair + (e & 1), j = mt * 16 + g + 8 * (e >> 1);
        if (f < n && d[nt][e] <= sh->limit[f]) sh->listed[atomicAdd(&sh->n_listed, 1)] = static_cast<uint16_t>(f * kEntries + j);
      }
    }
    __syncthreads();
    // ---- this block's candidates, exactly, one warp each; the smaller distance wins, on ties the lower index (argmin's rule)
    for (int c = warp; c < sh->n_listed; c += kWarps) {
      const int f = sh->listed[c] / kEntries, j = rank * kEntries + sh->listed[c] % kEntries;
      const float4* er = reinterpret_cast<const float4*>(a.books + (static_cast<size_t>(l) * kCodes + j) * kDim + lane * 8);
      const float4 u = __ldg(er), v = __ldg(er + 1);
      const float4* xr = reinterpret_cast<const float4*>(exact_x + f * kDim + lane * 8);
      const float4 xa = xr[0], xb = xr[1];
      const float ev[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w}, xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
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
                                                    : 0xfffffffeull << 32;
      if (lane == 0) atomicMin(&sh->best_in[f], key);
    }
    __syncthreads();
    {
      const int f = tid & 31, peer = tid >> 5;
      st_cluster_u64(map_to_cta(smem_u32(&sh->best[f][rank]), static_cast<uint32_t>(peer)), sh->best_in[f]);
    }
    cluster_sync_all();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int f = warp + kWarps * i;
      unsigned long long best = sh->best[f][lane & 15];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other < best ? other : best;
      }
      const bool none = best == ~0ull;                         // a residual that is not finite: no candidate
      const int j = none ? 0 : static_cast<int>(best & 0xffffffffu);
      if (rank == 0 && lane == 0 && f < n && !skip) {
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
    if (ensure_dynamic_smem(reinterpret_cast<const void*>(rvq_stack_kernel), rvqs::kSmemBytes) != 0 ||
        cudaFuncSetAttribute(rvq_stack_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      (void)cudaGetLastError();
      return -1;
    }
    return resident_clusters(rvq_stack_kernel, rvqs::kThreads, rvqs::kSmemBytes, rvqs::kCtas);
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
  return n_codes == rvqs::kCodes && rows <= static_cast<long long>(rvqs::kRows) * stack_slots();
}

int launch_rvq_stack(const RvqStack* stacks, int n_stacks, long long rows, float tau_rel, int* status, cudaStream_t st) {
  using namespace rvqs;
  if (n_stacks < 1 || n_stacks > 2 || !(tau_rel >= 0.f)) return -1;
  RvqStackArgs a = {};
  CUtensorMap maps[2];
  for (int i = 0; i < n_stacks; ++i) {
    const RvqStack& s = stacks[i];
    if (s.residual == nullptr || s.books16 == nullptr || s.books == nullptr || s.e_sq == nullptr || s.codes == nullptr) return -1;
    if ((reinterpret_cast<uintptr_t>(s.residual) | reinterpret_cast<uintptr_t>(s.books) | reinterpret_cast<uintptr_t>(s.books16)) & 15u) return -3;
    RvqStackArgs::Stack& d = a.stack[i];
    d.x = s.residual;
    d.books = s.books;
    d.e_sq = s.e_sq;
    d.codes = s.codes;
    d.layers = s.layers;
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
  const unsigned clusters = static_cast<unsigned>((rows + kRows - 1) / kRows);
  return launch_kernel(rvq_stack_kernel, dim3(clusters * kCtas, static_cast<unsigned>(n_stacks)), kThreads, kSmemBytes, st, kCtas, 0, maps[0], maps[1],
                       a, status);
}

}  // namespace fm
