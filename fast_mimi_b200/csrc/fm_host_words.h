// Device words (a status word, a call's error word) on their way to the host.  Host code only.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>
#include <mutex>

namespace fm {

// Pairs of host words that copies may land in.  They are a page of the library's own, page-locked on the first read, so that a
// copy does not block the caller and one wait serves two words; where the page cannot be locked, copies block and the words are
// read all the same.  A pair is a thread's for the time of one read; nothing is allocated and nothing grows.
class HostWords {
 public:
  HostWords() : pair_(take()) {}
  ~HostWords() {
    if (pair_ < kPairs) pool().used.fetch_and(~(1ull << pair_), std::memory_order_release);
  }
  HostWords(const HostWords&) = delete;
  HostWords& operator=(const HostWords&) = delete;
  int* data() { return pair_ < kPairs ? pool().words[pair_] : own_; }
  bool locked() const { return pair_ < kPairs && pool().locked.load(std::memory_order_acquire); }      // kernels may write them

 private:
  static constexpr int kPairs = 64;
  struct Pool {
    alignas(4096) int words[512][2];       // the page; the first kPairs of them
    alignas(4096) std::atomic<uint64_t> used;
    std::atomic<bool> locked;
    std::mutex locking;
  };
  static Pool& pool() {
    static Pool p{};                       // locked until the process ends
    return p;
  }
  static int take() {
    Pool& p = pool();
    if (!p.locked.load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> only_one(p.locking);
      if (!p.locked.load(std::memory_order_relaxed)) {
        // not to break a capture that another thread has under way
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        const bool relaxed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
        if (cudaHostRegister(p.words, sizeof(p.words), cudaHostRegisterPortable) == cudaSuccess)
          p.locked.store(true, std::memory_order_release);
        else
          (void)cudaGetLastError();
        if (relaxed) (void)cudaThreadExchangeStreamCaptureMode(&mode);
      }
    }
    uint64_t used = p.used.load(std::memory_order_relaxed);
    while (~used != 0) {
      const int free = __builtin_ctzll(~used);
      if (p.used.compare_exchange_weak(used, used | (1ull << free), std::memory_order_acquire, std::memory_order_relaxed)) return free;
    }
    return kPairs;                         // more threads than pairs: words of this call
  }
  const int pair_;
  int own_[2];
};

// Waits for `st` and reads the words at device addresses a and b, either of them null (read as 0), into words[2].
inline cudaError_t read_words(const int* a, const int* b, int* words, cudaStream_t st) {
  words[0] = words[1] = 0;
  if (a == nullptr && b == nullptr) return cudaStreamSynchronize(st);
  HostWords host;
  cudaError_t e = cudaSuccess;
  if (a != nullptr) e = cudaMemcpyAsync(host.data(), a, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess && b != nullptr) e = cudaMemcpyAsync(host.data() + 1, b, sizeof(int), cudaMemcpyDeviceToHost, st);
  // waited for whatever the copies returned: one under way must not land in words that are another call's by then
  const cudaError_t waited = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = waited;
  if (e != cudaSuccess) return e;
  if (a != nullptr) words[0] = host.data()[0];
  if (b != nullptr) words[1] = host.data()[1];
  return cudaSuccess;
}

}  // namespace fm
