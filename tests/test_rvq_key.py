"""Which entry a word of the few-vector search stands for (csrc/fm_rvq_key.h); no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_rvq_key.h"
#include <cstdio>
#include <cstring>
#include <initializer_list>
static unsigned long long key(float d, unsigned j) {
  unsigned bits;
  std::memcpy(&bits, &d, 4);
  return static_cast<unsigned long long>(bits) << 32 | j;
}
int main() {
  using namespace fm;
  for (int n : {1, 128, 2048}) {
    for (unsigned j : {0u, 1u, 127u, 2047u})
      for (float d : {0.f, 1e-30f, 3.f, 3e38f})
        if (rvq_entry_of(key(d, j), n) != (j < static_cast<unsigned>(n) ? static_cast<int>(j) : -1)) return std::printf("entry %u of %d\n", j, n), 1;
    if (rvq_entry_of(kRvqNoKey, n) != -1 || rvq_entry_of(kRvqNoCandidate, n) != -1 || rvq_entry_of(kRvqNotFinite, n) != 0) return std::printf("marks\n"), 1;
    // whatever shared memory holds: no word reaches past the codebook
    unsigned long long x = 88172645463325252ull;
    for (int i = 0; i < 2000000; ++i) {
      x ^= x << 13; x ^= x >> 7; x ^= x << 17;
      const int e = rvq_entry_of(x, n);
      if (e < -1 || e >= n) return std::printf("%llx -> %d of %d\n", x, e, n), 1;
    }
    for (unsigned low : {0x7fffffffu, 0x80000000u, 0xffffffffu, static_cast<unsigned>(n)})
      if (rvq_entry_of(low, n) != -1) return std::printf("low word %x of %d\n", low, n), 1;
  }
  if (!(key(3e38f, 2047) < kRvqNoCandidate && kRvqNoCandidate < kRvqNotFinite && kRvqNotFinite < kRvqNoKey)) return std::printf("order\n"), 1;
  return 0;
}
"""


def test_no_word_leads_out_of_the_codebook(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "key.cpp", tmp_path / "key"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
