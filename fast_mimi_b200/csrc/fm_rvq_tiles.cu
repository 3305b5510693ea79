// Residual vector quantisation of many vectors: all layers of one or two stacks in one kernel (sm_100a).  Same decisions as the
// chain of products and decision kernels in fm_rvq.cu (src/fast_mimi/model.py:2277-2291, :2408-2429).
//
// That chain is bound by what lies between its products: records (512 B a frame and layer) and residuals (FP32 and FP16, 2.5 KB)
// go through memory, and neither kernel's units are busy while the other runs.  Here a pair of blocks owns 256 vectors through
// their layers: FP32 residuals in tensor memory beside the accumulators, their FP16 copies, the products' A operand, in shared
// memory.  The codebooks stream past them, one entry per vector and layer is fetched in FP32, and nothing but codes is written.
// (Residuals in memory cost 384 KB of L2 traffic a layer and block, 15000 cycles; two tiles of 256 vectors a pair, in turn or side by
// side, leave no room for them on the chip.)
//
// A score has to cost little: 128 x 2048 of them a layer and block cross four schedulers while the tensor core makes them in 17400
// cycles.  So |e|^2 is part of the product (sixteen more columns of K: -|e|^2 / 2 in three FP16 parts against a power of two), and
// x.e - |e|^2 / 2 is only compared: the largest of 32 against the largest that the four threads of a vector have seen so far, and
// one by one only where eight of them come within the margin of that.  What does is listed, marked where the list is full, and decided at
// the end of the layer by exact FP32 distances.
//
// Of the 42000 cycles that a layer takes 24000 are scores, 4500 of them until the first are there (the tensor core issues for 18000; a
// thread looks at 64 scores in 2100, for 2176 of products), 3000 the candidates, 5500 the exact distances of the one vector in seven that
// has several, 9000 the new residuals (a thread reads a quarter of its vector's entry, sector by sector).
//
// Warps 0-15: scores, decisions, residuals.  Warp 16: codebooks.  Warp 17: MMA (leader block only).  Warps 18, 19: -|e|^2 / 2.
#include <math.h>

#include "fm_common.cuh"
#include "fm_kernels.h"
#include "fm_launch.h"
#include "fm_rvq_deal.h"

namespace fm {

namespace rvqt {
constexpr int kDim = 256, kBlockM = 128, kTileRows = 2 * kBlockM;
static_assert(kTileRows == RvqDeal::kTileRows, "what is dealt");
constexpr int kEpiWarps = 16, kThreads = (kEpiWarps + 4) * 32;
constexpr int kEpiRegs = 112, kIssueRegs = 32;
static_assert(512 * kEpiRegs + 128 * kIssueRegs <= kThreads * 96, "register pool of the launch");
constexpr int kEntries = 128, kShare = 64, kGroup = 32;        // of a step of products; of a thread's share of every other step; looked at at once
constexpr int kSlices = kDim / 64;                             // of 64 dimensions: of K, and of a vector, one for each of its four threads
constexpr int kChunkBytes = kBlockM * 128, kXBytes = kSlices * kChunkBytes;
constexpr int kSliceBytes = kEntries / 2 * 128;                // this block's half of a step's entries, one slice
constexpr int kStages = 3, kStageBytes = kSlices * kSliceBytes;
constexpr int kOnesBytes = kBlockM * 32, kTailBytes = kEntries / 2 * 32;       // sixteen more columns of K, rows of 32 bytes
constexpr int kTails = 4;
constexpr int kList = 8;                                       // candidates that a thread remembers
constexpr int kMany = 255;                                     // ... or more than that: the others are marked in `more`
constexpr int kWords = 2048 / kGroup;                          // of marks
constexpr int kBatch = 8, kBatchPitch = 1040;                  // of 32 vectors, how many are decided exactly at once; bytes from one to the next
constexpr int kMarks = 2 * kBatchPitch + 3 * 32;                // behind them
constexpr int kMaxLayers = 32;
constexpr int kTmemCols = 512, kResidual = 2 * kEntries;       // columns: two accumulators, then the residuals

struct Stack {
  float* x;                    // [rows, 256]: the vectors, overwritten with residuals where there is another layer
  const float* books;          // [layers, n_codes, 256]
  const float* e_sq;           // [layers, n_codes]
  long long* codes;            // [layers, rows]
  int layers;
  float e_max[kMaxLayers];
  float unit[kMaxLayers];      // power of two that -|e|^2 / 2 is a multiple of
};
struct Args {
  Stack stack[2];
  int rows, n_codes;
  float tau_rel;
  RvqDeal deal;
};

// What a pair works on: its tiles of the first stack, then those of the second, layer by layer.
struct Walk {
  int next, end, next1, end1;
  int stack, tile, layer, layers;
  bool alive;
  __device__ __forceinline__ Walk(const Args& a, int pair) {
    next = a.deal.first[0][pair];
    end = a.deal.first[0][pair + 1];
    next1 = a.deal.first[1][pair];
    end1 = a.deal.first[1][pair + 1];
    open(a);
  }
  __device__ __forceinline__ void open(const Args& a) {
    stack = next < end ? 0 : 1;
    alive = stack == 0 || next1 < end1;
    tile = stack == 0 ? next++ : next1++;
    layer = 0;
    layers = stack == 0 ? a.stack[0].layers : a.stack[1].layers;
  }
  __device__ __forceinline__ void step(const Args& a) {
    if (++layer == layers) open(a);
  }
};

struct Shared {
  uint64_t full[kStages], empty[kStages];      // full: in the leader, bytes of both blocks
  uint64_t acc_full[2], acc_empty[2];          // acc_empty: in the leader, the epilogue warps of both blocks
  uint64_t x_ready;                            // in the leader: both blocks' residuals are in place
  uint64_t tail_full[kTails], tail_empty[kTails];        // tail_full: in the leader, both blocks' -|e|^2 / 2 of a step
  uint32_t tmem_base, skip;
  CtaCtl ctl;
  Stack stack[2];
  alignas(16) float lead[kBlockM][4];          // largest scores of a vector's four threads so far
  alignas(16) float square[kBlockM][4];        // of a vector's four slices
  uint32_t list[kBlockM][4][kList];            // their candidates: a score, rounded up to 21 bits, and the entry
  alignas(4) uint8_t listed[kBlockM][4];
  uint16_t winner[kBlockM];                    // where distances decided
  uint32_t more[kWords][kBlockM];              // a bit an entry: a vector's candidates behind lists that are full (a word belongs to one of its threads)
};
constexpr int kSmemBytes = 1024 + kXBytes + kStages * kStageBytes + kOnesBytes + kTails * kTailBytes + static_cast<int>(sizeof(Shared));
static_assert(kSmemBytes <= 232448, "shared memory");

// Bar of the four warps that share a lane group of tensor memory, i.e. 32 vectors.
__device__ __forceinline__ void team_sync(int lg) {
  __syncwarp();
  asm volatile("bar.sync %0, 128;" ::"r"(lg + 1) : "memory");
}
__device__ __forceinline__ void warp_vote() {
  asm volatile("{\n\t.reg .b32 r;\n\t.reg .pred p;\n\tsetp.eq.u32 p, 0, 0;\n\tvote.sync.ballot.b32 r, p, 0xffffffff;\n\t}" ::: "memory");
}
__device__ __forceinline__ void load_global8(const float* p, float (&v)[8]) {      // one sector; p 32-byte aligned
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
// The sixteen columns' descriptor: rows of 32 bytes, 32-byte swizzle, eight rows are 256 bytes.
__device__ __forceinline__ uint64_t tail_desc(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(1) << 16) | (static_cast<uint64_t>(256 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(6) << 61);
}
// A score that is no smaller, in the upper 21 bits.
__device__ __forceinline__ uint32_t round_up(float v) {
  const uint32_t b = __float_as_uint(v);
  return ((b >> 31) != 0u ? b : b + 2047u) & ~2047u;
}
// A score as a number beyond kList, no smaller.
__device__ __forceinline__ uint32_t full(float v) {
  const uint32_t b = __float_as_uint(v);
  return b > kList ? b : kList + 1;
}
// Place i of a batch in a team's 4 KB of each chunk; eight places begin on different banks.
__device__ __forceinline__ uint8_t* staged(uint8_t* area, int i) { return area + (i >> 1) * (kChunkBytes + 32) + (i & 1) * kBatchPitch; }

// Residuals of a team's vectors into their places in `area` (this thread's slice; -1: not this one).
__device__ __forceinline__ void stage(uint8_t* area, int place, int q, uint32_t t_residual) {
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    uint32_t x[32];
    tmem_ld32(t_residual + part * 32, x);
    tmem_ld_wait();
    if (place >= 0) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(staged(area, place) + q * 256 + part * 128 + 16 * c) = make_uint4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
    }
  }
}

// Vectors whose lists are full have many candidates, and much the same ones (entries that are equal, or nearly).  So each entry that is one for
// any vector of the batch that is staged in `area` is read once, by one of the team's four warps, four of them at a time, and its distance from
// all of the batch found, added up as ever.  (18000 vectors x 8 layers, 9 entries of zero in every codebook 224 us, 40 263, 600 961; in the chain
// 284, 388 and 2340.  With one warp a vector and all 2048 entries as its candidates 7900, 10400 and 23600.)  Lane 8 * k + i keeps the nearest to
// vector i of the entries that came k-th.  Returns the code of the thread's vector, if it is one of `many`.  A function of its own: the loops
// over scores need all registers.
__device__ __noinline__ int decide_crowd(Shared* sh, uint8_t* area, const float* book, unsigned many, uint32_t t_residual, int n_steps) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lg = warp & 3, q = warp >> 2, row = lg * 32 + lane;
  uint32_t* marks = reinterpret_cast<uint32_t*>(area + kMarks);                            // [kWords]
  uint2* nearest = reinterpret_cast<uint2*>(area + kMarks + 4 * kWords);               // [warp of the team][kBatch]: distance, entry
  int code = 0;
#pragma unroll 1
  while (many != 0u) {
    unsigned rest = many;
#pragma unroll
    for (int i = 0; i < kBatch; ++i) rest &= rest - 1u;
    const unsigned batch = many ^ rest;
    const int place = (batch >> lane & 1u) != 0u ? __popc(batch & ((1u << lane) - 1u)) : -1;
    many = rest;
    stage(area, place, q, t_residual);
    if (q * 32 + lane < kWords) marks[q * 32 + lane] = 0u;
    team_sync(lg);
    if (place >= 0) {
      const int listed = sh->listed[row][q];
#pragma unroll 1
      for (int i = 0; i < (listed == kMany ? kList : listed); ++i) {
        const uint32_t j = sh->list[row][q][i] & 2047u;
        atomicOr(marks + j / kGroup, 1u << j % kGroup);
      }
#pragma unroll 1
      for (int i = q >> 1; listed == kMany && i < n_steps; i += 2) {
#pragma unroll 1
        for (int word = i * 4 + (q & 1) * 2; word < i * 4 + (q & 1) * 2 + 2; ++word)
          if (sh->more[word][row] != 0u) atomicOr(marks + word, sh->more[word][row]);
      }
    }
    team_sync(lg);
    // every fourth entry is this warp's
    const uint32_t own = 0x11111111u << q;
    unsigned words0 = __ballot_sync(0xffffffffu, (marks[lane] & own) != 0u), words1 = __ballot_sync(0xffffffffu, (marks[32 + lane] & own) != 0u);
    uint32_t word = 0u;
    int first = 0;
    auto next = [&]() {
      if (word == 0u) {
        if ((words0 | words1) == 0u) return -1;
        const int at = words0 != 0u ? __ffs(words0) - 1 : 31 + __ffs(words1);
        if (words0 != 0u) words0 &= words0 - 1u;
        else words1 &= words1 - 1u;
        word = marks[at] & own;
        first = at * kGroup;
      }
      const int j = first + __ffs(word) - 1;
      word &= word - 1u;
      return j;
    };
    float least = INFINITY;
    int win = 0;
#pragma unroll 1
    while ((word | words0 | words1) != 0u) {
      float e[4][8];
      int mine = -1;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = next();
        load_global8(book + static_cast<size_t>(j >= 0 ? j : 0) * kDim + 8 * lane, e[k]);
        if ((lane >> 3) == k) mine = j;
      }
#pragma unroll 1
      for (int i = 0; i < __popc(batch); ++i) {
        const float4* src = reinterpret_cast<const float4*>(staged(area, i)) + 2 * lane;
        const float4 xa = src[0], xb = src[1];
        const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
        float sum[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sum[k] = 0.f;
#pragma unroll
          for (int d = 0; d < 8; ++d) {
            const float diff = x[d] - e[k][d];
            sum[k] = fmaf(diff, diff, sum[k]);
          }
        }
        // each lane goes on with half of the entries until one is left
#pragma unroll
        for (int o = 16; o >= 8; o >>= 1) {
          const bool upper = (lane & o) != 0;
#pragma unroll
          for (int k = 0; k < o / 8; ++k) {
            const float keep = upper ? sum[k + o / 8] : sum[k], give = upper ? sum[k] : sum[k + o / 8];
            sum[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
        if ((lane & 7) == i && mine >= 0 && sum[0] < least) {        // entries come in ascending order
          least = sum[0];
          win = mine;
        }
      }
    }
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
      const float d = __shfl_xor_sync(0xffffffffu, least, o);
      const int j = __shfl_xor_sync(0xffffffffu, win, o);
      if (d < least || (d == least && j < win)) {          // ties go to the lower index (argmin's rule)
        least = d;
        win = j;
      }
    }
    if (lane < kBatch) nearest[q * kBatch + lane] = make_uint2(__float_as_uint(least), static_cast<uint32_t>(win));
    team_sync(lg);
    if (place >= 0) {
      uint2 best = nearest[place];
#pragma unroll
      for (int i = 1; i < 4; ++i) {
        const uint2 n = nearest[i * kBatch + place];
        const float d = __uint_as_float(n.x), d0 = __uint_as_float(best.x);
        if (d < d0 || (d == d0 && n.y < best.y)) best = n;
      }
      code = static_cast<int>(best.y);
    }
    team_sync(lg);                                 // before the area is written again
  }
  return code;
}
}  // namespace rvqt

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(rvqt::kThreads, 1)
rvq_tiles_kernel(const __grid_constant__ CUtensorMap tmap_books0, const __grid_constant__ CUtensorMap tmap_books1,
                 const __grid_constant__ rvqt::Args a, uint32_t idesc, int* status) {
  using namespace rvqt;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem_x = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_stage = smem_x + kXBytes;
  uint8_t* smem_ones = smem_stage + kStages * kStageBytes;     // the sixteen columns of A
  uint8_t* smem_tail = smem_ones + kOnesBytes;                 // and of B, of the steps in flight
  Shared* sh = reinterpret_cast<Shared*>(smem_tail + kTails * kTailBytes);
  CtaCtl* ctl = &sh->ctl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = rank == 0;
  const int pair = static_cast<int>(blockIdx.x >> 1);
  const int n_steps = a.n_codes / kEntries;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&sh->full[i], 1);
      mbar_init(&sh->empty[i], 1);
    }
    mbar_init(&sh->x_ready, 2 * kEpiWarps);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh->acc_full[i], 1);
      mbar_init(&sh->acc_empty[i], kEpiWarps);       // half of the warps of either block
    }
    for (int i = 0; i < kTails; ++i) {
      mbar_init(&sh->tail_full[i], 4);
      mbar_init(&sh->tail_empty[i], 1);
    }
    ctl->abort = 0;
    sh->skip = (status != nullptr && *reinterpret_cast<volatile int*>(status) != 0) ? 1u : 0u;
    fence_mbar_init();
  }
  for (int i = static_cast<int>(threadIdx.x); i < kTails * kTailBytes / 16; i += kThreads) reinterpret_cast<uint4*>(smem_tail)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
  if (threadIdx.x == 0) sh->stack[0] = a.stack[0];
  if (threadIdx.x == 32) sh->stack[1] = a.stack[1];
  if (warp == kEpiWarps) {
    tmem_alloc_pair(&sh->tmem_base, kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = sh->tmem_base;
  const bool skip = ld_shared_cluster_u32(map_to_cta(smem_u32(&sh->skip), 0)) != 0;

  if (skip) {
    // a kernel in front already reported an error through this status word: do nothing
  } else if (warp >= kEpiWarps) {
    warpgroup_reg_dec<kIssueRegs>();
    if (warp == kEpiWarps && lane == 0) {
      // ---------------------------------------------------------- codebooks
      tma_prefetch_desc(&tmap_books0);
      tma_prefetch_desc(&tmap_books1);
      int stage = 0;
      uint32_t phase = 0;
      for (Walk w(a, pair); w.alive; w.step(a)) {
        const CUtensorMap* map = w.stack == 0 ? &tmap_books0 : &tmap_books1;
        const int row0 = w.layer * a.n_codes + static_cast<int>(rank) * (kEntries / 2);
#pragma unroll 1
        for (int nt = 0; nt < n_steps; ++nt) {
          mbar_wait(&sh->empty[stage], phase ^ 1u, ctl, status, kErrWaitConsumer);
          if (leader) mbar_arrive_expect_tx(&sh->full[stage], 2 * kStageBytes);
#pragma unroll
          for (int kc = 0; kc < kSlices; ++kc)
            tma_load_2d_pair(smem_stage + stage * kStageBytes + kc * kSliceBytes, map, &sh->full[stage], kc * 64, row0 + nt * kEntries);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    } else if (warp == kEpiWarps + 1 && leader) {
      // ---------------------------------------------------------- products
      const bool elected = elect_one();
      const uint64_t x_desc = umma_desc_sw128(smem_u32(smem_x)), ones_desc = tail_desc(smem_u32(smem_ones));
      uint32_t step = 0, turn = 0, phase = 0;
      int stage = 0;
      for (Walk w(a, pair); w.alive; w.step(a), ++turn) {
        mbar_wait_cluster(&sh->x_ready, turn & 1u, ctl, status, kErrWaitConsumer);
#pragma unroll 1
        for (int nt = 0; nt < n_steps; ++nt, ++step) {
          const uint32_t buf = step & 1u, parity = (step >> 1) & 1u;
          mbar_wait(&sh->acc_empty[buf], parity ^ 1u, ctl, status, kErrWaitConsumer);
          tc_fence_after_sync();
          const uint32_t d_tmem = tmem_base + buf * kEntries;
          mbar_wait(&sh->full[stage], phase, ctl, status, kErrWaitTma);
          const uint32_t tail = step % kTails;
          mbar_wait_cluster(&sh->tail_full[tail], (step / kTails) & 1u, ctl, status, kErrWaitConsumer);
          warp_vote();                             // behind a wait alone the products would be issued half as fast
          tc_fence_after_sync();
          const uint64_t b_desc = umma_desc_sw128(smem_u32(smem_stage + stage * kStageBytes));
#pragma unroll
          for (int k = 0; k < 4 * kSlices; ++k)
            if (elected)
              tc_mma_ss_pair(d_tmem, x_desc + static_cast<uint64_t>((k / 4) * kChunkBytes >> 4) + 2u * (k % 4),
                             b_desc + static_cast<uint64_t>((k / 4) * kSliceBytes >> 4) + 2u * (k % 4), idesc, k != 0 ? 1u : 0u);
          // |e|^2 last: the tensor core cuts every addend to the accumulator's exponent
          if (elected) {
            tc_mma_ss_pair(d_tmem, ones_desc, tail_desc(smem_u32(smem_tail + tail * kTailBytes)), idesc, 1u);
            tc_commit_pair(&sh->acc_full[buf], 3);
            tc_commit_pair(&sh->empty[stage], 3);
            tc_commit_pair(&sh->tail_empty[tail], 3);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    } else if (warp >= kEpiWarps + 2) {
      // ---------------------------------------------------------- -|e|^2 / 2 of this block's half of a step's entries, one a thread
      const uint32_t tail_full_leader = map_to_cta(smem_u32(&sh->tail_full[0]), 0);
      const int r = (warp - kEpiWarps - 2) * 32 + lane;
      uint32_t step = 0;
      for (Walk w(a, pair); w.alive; w.step(a)) {
        const Stack& s = sh->stack[w.stack];
        const float* e_sq = s.e_sq + static_cast<size_t>(w.layer) * a.n_codes + rank * (kEntries / 2) + r;
        const float factor = -0.5f / s.unit[w.layer];
        float q = __ldg(e_sq);
#pragma unroll 1
        for (int nt = 0; nt < n_steps; ++nt, ++step) {
          const uint32_t tail = step % kTails;
          const float v = q * factor;
          if (nt + 1 < n_steps) q = __ldg(e_sq + (nt + 1) * kEntries);
          const __half hi = __float2half_rn(v);
          const float rest = v - __half2float(hi);
          const __half mid = __float2half_rn(rest), low = __float2half_rn(rest - __half2float(mid));
          mbar_wait(&sh->tail_empty[tail], ((step / kTails) & 1u) ^ 1u, ctl, status, kErrWaitConsumer);
          // the first eight of the row's sixteen columns (A is the same in both halves)
          *reinterpret_cast<uint2*>(smem_tail + tail * kTailBytes + r * 32 + (((r >> 2) & 1) << 4)) =
              make_uint2(__half_as_ushort(hi) | (static_cast<uint32_t>(__half_as_ushort(mid)) << 16), __half_as_ushort(low));
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(tail_full_leader + tail * 8u);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ scores, decisions, residuals
    warpgroup_reg_inc<kEpiRegs>();
    // This thread's vector, its slice of the vector's dimensions, and its share of the entries: one half of every other step.
    const int lg = warp & 3, q = warp >> 2, row = lg * 32 + lane;
    const uint32_t acc_empty_leader = map_to_cta(smem_u32(&sh->acc_empty[0]), 0);
    const uint32_t x_ready_leader = map_to_cta(smem_u32(&sh->x_ready), 0);
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(lg * 32) << 16), t_residual = t_row + kResidual + q * 64;
    auto vector = [&](int tile) { return static_cast<long long>(tile) * kTileRows + static_cast<int>(rank) * kBlockM + row; };
    // 32 dimensions of the thread's slice enter a layer: in FP32, in FP16, and their squares.
    auto enter = [&](int part, const float (&x)[32], float& square) {
#pragma unroll
      for (int k = 0; k < 32; ++k) square = fmaf(x[k], x[k], square);
      uint32_t bits[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) bits[k] = __float_as_uint(x[k]);
      tmem_st32(t_residual + part * 32, bits);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4*>(smem_x + q * kChunkBytes + sw128_offset(static_cast<uint32_t>(row), static_cast<uint32_t>(part * 4 + c))) =
            make_uint4(Pack16<__half>::pack(x[8 * c], x[8 * c + 1]), Pack16<__half>::pack(x[8 * c + 2], x[8 * c + 3]),
                       Pack16<__half>::pack(x[8 * c + 4], x[8 * c + 5]), Pack16<__half>::pack(x[8 * c + 6], x[8 * c + 7]));
    };
    auto publish = [&](float square, float unit) {
      sh->square[row][q] = square;
      sh->lead[row][q] = -INFINITY;
      if (q < 2)                                   // this thread's eight of A's sixteen more columns
        *reinterpret_cast<uint4*>(smem_ones + row * 32 + q * 16) = make_uint4(Pack16<__half>::pack(unit, unit), Pack16<__half>::pack(unit, 0.f), 0u, 0u);
      tmem_st_wait();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(x_ready_leader);
      team_sync(lg);
    };
    auto begin_task = [&](const Walk& w) {
      const Stack& s = sh->stack[w.stack];
      const long long v = vector(w.tile);
      float square = 0.f;
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {
        float x[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) x[k] = 0.f;
        if (v < a.rows) {
          const float4* src = reinterpret_cast<const float4*>(s.x + v * kDim + q * 64 + part * 32);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float4 f = __ldcg(src + k);
            x[4 * k] = f.x; x[4 * k + 1] = f.y; x[4 * k + 2] = f.z; x[4 * k + 3] = f.w;
          }
        }
        enter(part, x, square);
      }
      publish(square, s.unit[0]);
    };

    uint32_t use = 0;                              // of this thread's accumulator
    const uint32_t buf = static_cast<uint32_t>(q >> 1);
    Walk w(a, pair);
    if (w.alive) begin_task(w);
#pragma unroll 1
    while (w.alive) {
      const Stack& s = sh->stack[w.stack];
      const int layer = w.layer;
      // The margin of the vector (fm_rvq.cu), halved as scores are half the distances, and what the tensor core cuts off beside
      // |e|^2 / 2.  (It keeps addends down to 2^-25 of the largest one's power of two and cuts the result to 24 bits, as 1 - 1 + 2^-k shows.  In the
      // last instruction the sum x.e and the least of the three parts lose less than 2^-25 of M, the larger of |x.e| and |e|^2 / 2, each, the
      // result, which is less than 2 M, 2^-22 M, and |e|^2 was rounded by 2^-24: together 1.5 * 2^-22 M, of two scores at M = |e|^2 / 2
      // 1.5 * 2^-22 |e|^2.  Taken: 2^-21.  For a larger M, and for the sixteen instructions before, 3e-5 |x||e| is in what tau_rel has to spare.)
      // Where the vector is not finite, or none, nothing is a candidate.
      float margin;
      {
        const float4 sq = *reinterpret_cast<const float4*>(sh->square[row]);
        const float e_max = s.e_max[layer];
        margin = 0.5f * (rvq_margin((sq.x + sq.y) + (sq.z + sq.w), e_max, a.tau_rel) + 9.5367431640625e-7f * e_max * e_max);
        if (!(margin < INFINITY) || vector(w.tile) >= a.rows) margin = NAN;
      }
      // ---- the scores of this thread's entries
      uint32_t n = 0u;                             // of them in its list; beyond kList: it is full, and the largest of what it remembers
      {
        uint32_t* list = sh->list[row][q];
        volatile float* known = sh->lead[row];
        float best = -INFINITY;
#pragma unroll 1
        for (int nt = static_cast<int>(buf); nt < n_steps; nt += 2, ++use) {
          // what the other three know is as good a bound, however old
          float lead = fmaxf(max3(known[0], known[1], known[2]), fmaxf(known[3], best));
          mbar_wait(&sh->acc_full[buf], use & 1u, ctl, status, kErrWaitMma);
          tc_fence_after_sync();
          // both groups of 32 at once, so that the accumulator is free again before they are looked at
          uint32_t scores[kShare / kGroup][kGroup];
#pragma unroll
          for (int part = 0; part < kShare / kGroup; ++part)
            tmem_ld32(t_row + buf * kEntries + static_cast<uint32_t>((q & 1) * kShare + part * kGroup), scores[part]);
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(acc_empty_leader + buf * 8u);
#pragma unroll
          for (int part = 0; part < kShare / kGroup; ++part) {
            const uint32_t(&raw)[kGroup] = scores[part];
            float m[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t* r = raw + 8 * j;
              m[j] = max3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
              m[j] = max3(m[j], __uint_as_float(r[3]), __uint_as_float(r[4]));
              m[j] = max3(m[j], __uint_as_float(r[5]), __uint_as_float(r[6]));
              m[j] = fmaxf(m[j], __uint_as_float(r[7]));
            }
            const float top = fmaxf(max3(m[0], m[1], m[2]), m[3]);
            const bool near = top >= lead - margin;
            lead = fmaxf(lead, top);
            best = fmaxf(best, top);
            if (__any_sync(0xffffffffu, near)) {
              const float limit = near ? top - margin : NAN;         // of this group's entries
              uint32_t mask = 0u;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (__any_sync(0xffffffffu, m[j] >= limit)) {
#pragma unroll
                  for (int c = 8 * j; c < 8 * j + 8; ++c)
                    if (__uint_as_float(raw[c]) >= limit) mask |= 1u << c;
                }
              }
              const uint32_t key = round_up(top) | static_cast<uint32_t>(nt * kEntries + (q & 1) * kShare + part * kGroup);
              for (; mask != 0u; mask &= mask - 1u) {
                if (n >= kList) {
                  if (n > kList) {                 // entries are marked; if all that it remembers is out of reach by now, it begins anew
                    if (lead - margin > __uint_as_float(n)) n = 0u;
                  } else {                         // those that are out of reach by now go, or they stay in the list and what comes is marked
                    n = 0u;
                    float most = -INFINITY;
#pragma unroll 1
                    for (int i = 0; i < kList; ++i) {
                      const uint32_t old = list[i];
                      const float score = __uint_as_float(old & ~2047u);
                      most = fmaxf(most, score);
                      if (score >= lead - margin) list[n++] = old;
                    }
                    if (n == kList) {
                      n = full(most);
#pragma unroll 1
                      for (int i = static_cast<int>(buf); i < n_steps; i += 2)
                        sh->more[i * 4 + (q & 1) * 2][row] = sh->more[i * 4 + (q & 1) * 2 + 1][row] = 0u;
                    }
                  }
                  if (n > kList) {
                    sh->more[nt * 4 + (q & 1) * 2 + part][row] = mask;
                    n = full(fmaxf(top, __uint_as_float(n)));
                    break;
                  }
                }
                list[n++] = key + static_cast<uint32_t>(__ffs(mask) - 1);
              }
              __syncwarp();
            }
          }
          known[q] = best;
        }
      }
      team_sync(lg);
      // ---- the decision; every entry that is within the margin of the largest score of all four threads
      const bool last = layer + 1 == w.layers;
      const long long v = vector(w.tile);
      const float* book = s.books + static_cast<size_t>(layer) * a.n_codes * kDim;
      int code = 0;
      {
        const float4 l = *reinterpret_cast<const float4*>(sh->lead[row]);
        const float limit = fmaxf(max3(l.x, l.y, l.z), l.w) - margin;
        int kept_here = 0;
        if (n <= kList) {
          for (int i = 0; i < static_cast<int>(n); ++i) {
            const uint32_t key = sh->list[row][q][i];
            if (__uint_as_float(key & ~2047u) >= limit) sh->list[row][q][kept_here++] = key;
          }
        } else if (__uint_as_float(n) >= limit) {
          kept_here = kMany;
        }
        sh->listed[row][q] = static_cast<uint8_t>(kept_here);
        team_sync(lg);
        const uchar4 kept = *reinterpret_cast<const uchar4*>(sh->listed[row]);
        const int all = kept.x + kept.y + kept.z + kept.w;
        if (all == 0 && q == 0 && v < a.rows && status != nullptr) atomicMax(status, static_cast<int>(kErrNonFinite));     // not finite
        if (all == 1) code = static_cast<int>(sh->list[row][kept.x != 0 ? 0 : (kept.y != 0 ? 1 : (kept.z != 0 ? 2 : 3))][0] & 2047u);       // the only candidate has won
        // The others' residuals cross shared memory, a few vectors at a time, where the team's FP16 copies lay (their products are
        // complete), and a warp takes a vector: its candidates' distances, added up as in fm_rvq.cu.  (The four warps come to the same
        // rounds.)
        const unsigned many = __ballot_sync(0xffffffffu, kept.x == kMany || kept.y == kMany || kept.z == kMany || kept.w == kMany);
        uint8_t* area = smem_x + lg * (32 * 128);
#pragma unroll 1
        for (unsigned open = __ballot_sync(0xffffffffu, all > 1) & ~many; open != 0u;) {
          unsigned rest = open;
#pragma unroll
          for (int i = 0; i < kBatch; ++i) rest &= rest - 1u;
          const unsigned batch = open ^ rest;
          const int place = __popc(batch & ((1u << lane) - 1u));
          const bool mine = (batch >> lane & 1u) != 0u;
          stage(area, mine ? place : -1, q, t_residual);
          team_sync(lg);
#pragma unroll 1
          for (int i = q; i < __popc(batch); i += 4) {
            unsigned behind = batch;
            for (int k = 0; k < i; ++k) behind &= behind - 1u;
            const int r = lg * 32 + __ffs(behind) - 1;
            const uchar4 count = *reinterpret_cast<const uchar4*>(sh->listed[r]);
            const int entries = count.x + count.y + count.z + count.w;
            // lane k * kList + i: place i of thread k's list
            const uint32_t key = sh->list[r][lane / kList][lane % kList];
            unsigned keys = __ballot_sync(0xffffffffu, lane % kList < sh->listed[r][lane / kList]);
            const float4* src = reinterpret_cast<const float4*>(staged(area, i)) + 2 * lane;
            const float4 xa = src[0], xb = src[1];
            const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
            float least = INFINITY;
            int win = 0;
#pragma unroll 1
            for (int c = 0; c < entries; c += 4) {
              float e[4][8], sum[4];
              int j[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int from = __shfl_sync(0xffffffffu, static_cast<int>(key & 2047u), (__ffs(keys) - 1) & 31);
                keys &= keys - 1u;
                j[k] = c + k < entries ? from : -1;
                // not under a test: e would be alive all through the kernel (18000 vectors x 8 layers 189 us instead of 180)
                load_global8(book + static_cast<size_t>(j[k] >= 0 ? j[k] : 0) * kDim + 8 * lane, e[k]);
              }
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                sum[k] = 0.f;
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                  const float diff = x[d] - e[k][d];
                  sum[k] = fmaf(diff, diff, sum[k]);
                }
              }
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                for (int k = 0; k < 4; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
              }
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (j[k] >= 0 && (sum[k] < least || (sum[k] == least && j[k] < win))) {      // ties go to the lower index (argmin's rule)
                  least = sum[k];
                  win = j[k];
                }
              }
            }
            if (lane == 0) sh->winner[r] = static_cast<uint16_t>(win);
          }
          team_sync(lg);
          if (mine) code = sh->winner[row];
          open = rest;
        }
        if (many != 0u) {
          const int found = decide_crowd(sh, area, book, many, t_residual, n_steps);
          if ((many >> lane & 1u) != 0u) code = found;
        }
        if (q == 0 && v < a.rows) s.codes[static_cast<long long>(layer) * a.rows + v] = code;
      }
      // ---- the new residuals
      if (!last) {
        float square = 0.f;
#pragma unroll 1
        for (int part = 0; part < 2; ++part) {
          uint32_t bits[32];
          tmem_ld32(t_residual + part * 32, bits);
          float e[4][8];
#pragma unroll
          for (int c = 0; c < 4; ++c) load_global8(book + static_cast<size_t>(code) * kDim + q * 64 + part * 32 + 8 * c, e[c]);
          tmem_ld_wait();
          float x[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = v < a.rows ? __uint_as_float(bits[i]) - e[i >> 3][i & 7] : 0.f;
          enter(part, x, square);
        }
        publish(square, s.unit[layer + 1]);
      }
      w.step(a);
      if (w.alive && last) begin_task(w);
    }
  }

  // Neither block may leave (or release tensor memory) while its partner can still signal it.
  tc_fence_before_sync();
  __syncthreads();
  if (ctl->abort) __nanosleep(20000);   // copies that may still be in flight get time to land
  cluster_sync_all();
  if (warp == kEpiWarps) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

namespace {
// What the kernel needs of its stacks: -|e|^2 / 2 has to fit FP16 times the largest power of two that FP16 holds, and entries are read
// by whole sectors.  0, -1, or -3 for an address.
int cannot(const RvqStack* stacks, int n_stacks, long long rows, int n_codes) {
  using namespace rvqt;
  if (n_stacks < 1 || n_stacks > 2 || rows < 0 || rows > 0x7fffffffLL || n_codes <= 0 || n_codes % (2 * kEntries) != 0 || n_codes > 2048) return -1;
  int rc = 0;
  for (int i = 0; i < n_stacks; ++i) {
    const RvqStack& s = stacks[i];
    if (s.residual == nullptr || s.books16 == nullptr || s.books == nullptr || s.e_sq == nullptr || s.e_max == nullptr || s.codes == nullptr ||
        s.layers < 1 || s.layers > kMaxLayers)
      return -1;
    for (int l = 0; l < s.layers; ++l)
      if (!(s.e_max[l] >= 0.f && s.e_max[l] <= 16384.f)) return -1;
    if (((reinterpret_cast<uintptr_t>(s.residual) | reinterpret_cast<uintptr_t>(s.books16) | reinterpret_cast<uintptr_t>(s.e_sq)) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(s.books) & 31u) != 0)
      rc = -3;
  }
  return rc;
}
}  // namespace

static RvqDeal deal_stacks(const RvqStack* stacks, int n_stacks, long long rows) {
  const int l0 = stacks[0].layers, l1 = n_stacks == 2 ? stacks[1].layers : 0;
  RvqDeal deal;
  deal.make(rows, l0 > l1 ? l0 : l1, l0 > l1 ? l1 : l0 * (n_stacks - 1), sm_count());
  return deal;
}

bool rvq_tiles_take(const RvqStack* stacks, int n_stacks, long long rows, int n_codes) {
  return cannot(stacks, n_stacks, rows, n_codes) == 0 && rows > 0 && rvq_tiles_pay(deal_stacks(stacks, n_stacks, rows), rows, n_codes);
}

int launch_rvq_tiles(const RvqStack* stacks, int n_stacks, long long rows, int n_codes, float tau_rel, int* status, cudaStream_t st) {
  using namespace rvqt;
  if (!(tau_rel >= 0.f)) return -1;
  int rc = cannot(stacks, n_stacks, rows, n_codes);
  if (rc != 0 || rows == 0) return rc;
  Args a = {};
  CUtensorMap maps[2];
  const int longer = n_stacks == 2 && stacks[1].layers > stacks[0].layers ? 1 : 0;
  for (int i = 0; i < n_stacks; ++i) {
    const RvqStack& s = stacks[i ^ longer];
    Stack& d = a.stack[i];
    d.x = s.residual;
    d.books = s.books;
    d.e_sq = s.e_sq;
    d.codes = s.codes;
    d.layers = s.layers;
    for (int l = 0; l < s.layers; ++l) {
      d.e_max[l] = s.e_max[l];
      int exponent = 0;                        // -|e|^2 / 2 in units of the least power of two that keeps it below 2^14
      frexpf(0.5f * s.e_max[l] * s.e_max[l], &exponent);
      exponent -= 14;
      d.unit[l] = ldexpf(1.f, exponent < -14 ? -14 : (exponent > 15 ? 15 : exponent));
    }
    rc = encode_rows_16bit(&maps[i], s.books16, static_cast<uint64_t>(s.layers) * n_codes, kDim, kEntries / 2, 64);
    if (rc != 0) return rc;
  }
  if (n_stacks == 1) maps[1] = maps[0];
  a.rows = static_cast<int>(rows);
  a.n_codes = n_codes;
  a.tau_rel = tau_rel;
  a.deal = deal_stacks(stacks, n_stacks, rows);
  const uint32_t idesc = umma_idesc_f16(kTileRows, kEntries, 0, 0, 0, 0);
  rc = ensure_dynamic_smem(reinterpret_cast<const void*>(rvq_tiles_kernel), kSmemBytes);
  if (rc != 0) return rc;
  return launch_kernel(rvq_tiles_kernel, dim3(static_cast<unsigned>(2 * a.deal.pairs)), kThreads, kSmemBytes, st, 1, 0, maps[0], maps[1], a, idesc, status);
}

}  // namespace fm
