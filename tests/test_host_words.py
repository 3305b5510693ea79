"""How error words reach the host (csrc/fm_host_words.h), against a stand-in for the CUDA runtime: no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_host_words.h"
#include <cstdio>
#include <cstring>
#include <set>
#include <thread>
#include <vector>

// The stand-in: device words are host words, a copy lands when the stream is waited for.
static std::atomic<int> n_registered{0}, n_allocated{0};
static bool can_register = true;
static int copies_left = 1 << 30;
struct Copy { void* to; const void* from; size_t bytes; };
static thread_local std::vector<Copy> under_way;
static thread_local int n_waits = 0;
extern "C" {
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
  if (reinterpret_cast<uintptr_t>(p) % 4096 != 0 || n % 4096 != 0) return cudaErrorInvalidValue;
  if (!can_register) return cudaErrorMemoryAllocation;
  ++n_registered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void**, size_t, unsigned) { ++n_allocated; return cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (copies_left-- <= 0) return cudaErrorInvalidValue;
  under_way.push_back({to, from, n});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  ++n_waits;
  for (const Copy& c : under_way) std::memcpy(c.to, c.from, c.bytes);
  under_way.clear();
  return cudaSuccess;
}
}

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  int words[2] = {9, 9};
  const int a = 101, b = 7;
  can_register = false;                                  // no page-locked memory: the words are read all the same
  CHECK(fm::read_words(&a, &b, words, nullptr) == cudaSuccess && words[0] == 101 && words[1] == 7);
  can_register = true;
  for (int i = 0; i < 3; ++i) CHECK(fm::read_words(&a, &b, words, nullptr) == cudaSuccess && words[0] == 101 && words[1] == 7);
  CHECK(n_registered == 1 && n_waits == 4);              // asked for again, then kept; one wait a call
  CHECK(fm::read_words(nullptr, &b, words, nullptr) == cudaSuccess && words[0] == 0 && words[1] == 7);
  CHECK(fm::read_words(&a, nullptr, words, nullptr) == cudaSuccess && words[0] == 101 && words[1] == 0);
  CHECK(fm::read_words(nullptr, nullptr, words, nullptr) == cudaSuccess && words[0] == 0 && words[1] == 0);
  copies_left = 1;                                       // the second copy fails: the first is waited for, nothing is handed out
  CHECK(fm::read_words(&a, &b, words, nullptr) == cudaErrorInvalidValue && words[0] == 0 && words[1] == 0 && under_way.empty());
  copies_left = 1 << 30;
  {                                                      // no two reads under way share words, however many there are
    std::vector<std::unique_ptr<fm::HostWords>> held;
    std::set<int*> places;
    for (int i = 0; i < 200; ++i) {
      held.push_back(std::make_unique<fm::HostWords>());
      places.insert(held.back()->data());
    }
    CHECK(places.size() == 200);
  }
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 100; ++t)
    threads.emplace_back([t, &wrong] {
      const int mine[2] = {1000 + t, 2000 + t};
      for (int i = 0; i < 300; ++i) {
        int got[2];
        if (fm::read_words(&mine[0], &mine[1], got, nullptr) != cudaSuccess || got[0] != mine[0] || got[1] != mine[1]) ++wrong;
      }
    });
  for (auto& t : threads) t.join();
  CHECK(wrong == 0 && n_registered == 1 && n_allocated == 0);
  std::puts("ok");
  return 0;
}
"""


def test_error_words_are_read_whether_or_not_memory_can_be_locked(tmp_path):
    from fast_mimi_b200 import _build
    cxx = os.environ.get("CXX") or shutil.which("g++")
    include = os.path.join(os.path.dirname(os.path.dirname(_build.find_nvcc())), "include")
    if cxx is None or not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no C++ compiler or CUDA headers here")
    source, program = tmp_path / "words.cpp", tmp_path / "words"
    source.write_text("#include <memory>\n" + PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), "-I", include, str(source), "-o",
                    str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout + done.stderr
