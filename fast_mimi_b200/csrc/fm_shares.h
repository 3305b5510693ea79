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

}  // namespace fm
