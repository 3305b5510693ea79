// A candidate of the search of few vectors (fm_rvq_stack.cu) as one word, (distance << 32 | index): the smallest wins, on ties the lower index.
// Host and device code.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define FM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FM_HOST_DEVICE inline
#endif

namespace fm {

constexpr unsigned long long kRvqNoKey = ~0ull;                              // nothing yet
constexpr unsigned long long kRvqNotFinite = 0xfffffffeull << 32;            // an exact distance that is not finite: above those that are, index 0
constexpr unsigned long long kRvqNoCandidate = 0xfffffffdull << 32;          // approximate distances that are not: no entry, whatever the others find

// The entry that a key stands for, -1 for none.  Never outside the codebook: after a wait that gave up (the kernel ends with a status word) the key is
// whatever lay in shared memory, and the entry is read all the same.
FM_HOST_DEVICE int rvq_entry_of(unsigned long long key, int n_codes) {
  const uint32_t index = static_cast<uint32_t>(key);
  return key == kRvqNoCandidate || index >= static_cast<uint32_t>(n_codes) ? -1 : static_cast<int>(index);
}

}  // namespace fm

#undef FM_HOST_DEVICE
