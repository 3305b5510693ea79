"""How the steps of a persistent kernel are dealt out to its blocks (csrc/fm_shares.h); no GPU needed."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "fm_shares.h"
#include <initializer_list>
#include <cstdio>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (sequences %d of %d tiles, %d blocks)\n", __LINE__, #x, seqs, tiles, blocks); return 1; } } while (0)
int main() {
  for (int blocks : {1, 2, 7, 132, 148})
    for (int seqs = 8; seqs <= 400; seqs += 8)
      for (int tiles : {3, 4, 5, 8, 12, 20, 79}) {
        const int n = seqs * tiles;
        const fm::Shares s(n, blocks);
        const int used = s.used();
        CHECK(used >= 1 && used <= blocks && used <= n && s.first(0) == 0 && s.first(used) == n);
        CHECK(fm::Shares(n, used).per_block == s.per_block);                   // the kernel, which has the number of its blocks, deals alike
        CHECK(s.per_block == (n + blocks - 1) / blocks);                       // no block could have fewer
        for (int b = 0; b < used; ++b) CHECK(s.first(b + 1) > s.first(b) && s.first(b + 1) - s.first(b) <= s.per_block);
        // where a share is a whole number of sequences or a whole part of one, none begins inside of a sequence but at such a part
        if (s.per_block % tiles == 0) for (int b = 0; b < used; ++b) CHECK(s.first(b) % tiles == 0);
        if (tiles % s.per_block == 0) for (int b = 0; b < used; ++b) CHECK(s.first(b) / tiles == (s.first(b + 1) - 1) / tiles);
      }
  const int seqs = 0, tiles = 0, blocks = 148;
  CHECK(fm::Shares(0x7fffffff, 148).first(148) == 0x7fffffff && fm::Shares(0x7fffffff, 148).first(147) < 0x7fffffff);
  std::puts("ok");
  return 0;
}
"""


def test_shares_cover_every_step_and_keep_to_sequences(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler here")
    source, program = tmp_path / "shares.cpp", tmp_path / "shares"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fast_mimi_b200", "csrc"), str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0 and done.stdout.strip() == "ok", done.stdout
