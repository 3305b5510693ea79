// A chain of steps dealt out to the blocks of a persistent kernel.
#pragma once

#ifdef __CUDACC__
#define FM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FM_HOST_DEVICE inline
#endif

namespace fm {

// Block b of `blocks` takes steps [first(b), first(b + 1)): as few per block as fit on that many, the same number in all but the last.
// (So a share whose length divides a sequence's, or is a multiple of it, never begins inside of one by chance.)
struct Shares {
  int n_steps, per_block;
  FM_HOST_DEVICE Shares(int n_steps_, int blocks) : n_steps(n_steps_), per_block(static_cast<int>((n_steps_ + (blocks - 1ll)) / blocks)) {}
  FM_HOST_DEVICE int first(int block) const {
    const long long at = static_cast<long long>(block) * per_block;
    return at < n_steps ? static_cast<int>(at) : n_steps;
  }
  // Blocks that get any: dealt out to these, the shares are the same.
  FM_HOST_DEVICE int used() const { return static_cast<int>((n_steps + (per_block - 1ll)) / per_block); }
};

}  // namespace fm
