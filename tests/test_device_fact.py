"""What is kept of a device (csrc/fm_device_fact.h); no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_device_fact.h"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  static fm::DeviceFact fact;
  int asked = 0;
  auto fails = [&] { ++asked; return -1; };
  auto says = [&](int n) { return [&asked, n] { ++asked; return n; }; };
  CHECK(fact.get(3, fails) == -1 && fact.get(3, fails) == -1 && asked == 2);          // a failure is not kept
  CHECK(fact.get(3, says(7)) == 7 && fact.get(3, fails) == 7 && asked == 3);          // an answer is
  CHECK(fact.get(2, says(0)) == 0 && fact.get(2, fails) == 0 && asked == 4);          // none at all is an answer too, and devices have their own
  CHECK(fact.get(64, says(5)) == 5 && fact.get(64, says(6)) == 6 && fact.get(-1, says(1)) == 1);      // devices beyond the table are asked each time
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&] {
      for (int i = 0; i < 2000; ++i)
        for (int d = 8; d < 64; ++d)
          if (fact.get(d, [d] { return 100 + d; }) != 100 + d) ++wrong;
    });
  for (auto& t : threads) t.join();
  CHECK(wrong == 0);
  std::puts("ok");
  return 0;
}
"""


def test_answers_are_kept_and_failures_are_not(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "fact.cpp", tmp_path / "fact"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)],
                   check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout
