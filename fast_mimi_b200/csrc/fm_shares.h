// The steps of sequences of equal length dealt out to the blocks of a persistent kernel.
#pragma once

#ifdef __CUDACC__
#define FM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FM_HOST_DEVICE inline
#endif

namespace fm {

// No block has more steps than the fewest that the largest share can have.  Where that leaves room for it every sequence is cut
// alike and no share goes on into a second one; else the shares run on from sequence to sequence, all but the last of that length, so
// that one which is a whole number of sequences begins where one begins.  Worked out on the host: the divisions cost a kernel of
// 9 us 0.4 us.
struct Shares {
  int n_steps = 0, tiles = 1, per_block = 1, cuts = 0;       // cuts: shares of a sequence, 0 where they run on
  Shares() = default;
  Shares(int n_seqs, int tiles_, int blocks) : n_steps(n_seqs * tiles_), tiles(tiles_), per_block(up(n_steps, blocks)), cuts(up(tiles_, per_block)) {
    if (static_cast<long long>(n_seqs) * cuts > blocks) cuts = 0;
  }
  int used() const { return cuts > 0 ? n_steps / tiles * cuts : up(n_steps, per_block); }      // blocks that get any
  // Share of block `block` < used(): its first step, as a sequence and the tile of it, and its length.
  FM_HOST_DEVICE void share(int block, int* seq, int* tile, int* steps) const {
    int rest;
    if (cuts > 0) {
      *seq = block / cuts;
      *tile = (block - *seq * cuts) * per_block;
      rest = tiles - *tile;
    } else {
      const int at = block * per_block;
      *seq = at / tiles;
      *tile = at - *seq * tiles;
      rest = n_steps - at;
    }
    *steps = rest < per_block ? rest : per_block;
  }

 private:
  static int up(int a, int b) { return static_cast<int>((static_cast<long long>(a) + b - 1) / b); }
};

// Whether clips' heads (fm_fused_clip.cu), dealt evenly to `pairs` of blocks, are out sooner than whole clips in turn.  A dealt head costs up to a tenth
// more: a clip that two pairs share is loaded twice, and the warps that look up whose head is next have no registers left.  Calls on new inputs,
// whole -> dealt, us, by heads a pair:  8 -> 1 42.6 -> 19.2, 8 -> 7 44.2 -> 43.0, 16 -> 14 80.6 -> 78.9, 16 -> 15 84.1 -> 85.1, 24 -> 22 119.7 -> 120.5, 24 -> 23 126.6 -> 129.7,
// 32 -> 29 157.5 -> 156.5, 32 -> 30 162.0 -> 163.5, 32 -> 31 163.9 -> 169.1, 40 -> 37 200.6 -> 201.6, 48 -> 45 236.9 -> 239.5, 56 -> 51 277.0 -> 274.2, 56 -> 53 285.1 -> 289.3,
// 56 -> 55 288.1 -> 297.7 (in a captured graph, over and over on one input, dealing gains some two percent more: 24 -> 22 112.8 -> 109.0, 56 -> 53 247.9 -> 247.6).
inline bool dealt_heads_pay(const Shares& shares, int clips, int pairs) {
  const long long whole = 8ll * ((clips + pairs - 1ll) / pairs);
  return 12ll * shares.per_block < 11 * whole;
}

}  // namespace fm
